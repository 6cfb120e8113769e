"""Edges of the row-walking kernels: how live rows are found (one warp's registers, a prefix in shared memory, slot by
slot), rows cut into pieces, 32-byte and 16-byte aligned sources, plans below and above the ranking table's expert
limit, ragged compressor tiles, idle experts and the K split of the narrow GEMM, SiTU against 64 bits."""
import numpy as np
import pytest
import torch

from oracle import paired_nvfp4_oracle as orc
from helpers import bf16_tensor, bf16_bits, u8, dev, make_acts

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    import paired_nvfp4_kernels  # noqa: F401
    return torch.ops.paired_nvfp4


ROWS_CASES = [
    # E, cap, K, counts ("rand" or a list; out-of-range counts are clamped), offset of x in elements
    (1, 3, 7168, [3], 0),                 # one expert, a row in seven pieces
    (8, 16, 4096, [1, 0, 16, -3, 99, 5, 0, 2], 0),
    (32, 5, 1056, "rand", 8),             # as many experts as a warp holds, KB = 33: one block past a step; 16-byte aligned
    (33, 40, 96, "rand", 0),              # prefix in shared memory, KB = 3: scale words with slop
    (300, 130, 256, "rand", 8),           # several rounds of the block's scan, two row atoms
    (8200, 2, 32, "rand", 0),             # more experts than the prefix holds
    (40, 700, 1024, "rand", 0),           # more rows than warps
]


@pytest.mark.parametrize("E,cap,K,counts,offset", ROWS_CASES)
def test_quant_act_and_planned_scatter(ops, E, cap, K, counts, offset):
    rng = np.random.default_rng(E + K)
    cnt = rng.integers(0, cap + 1, E).astype(np.int32) if isinstance(counts, str) else np.array(counts, np.int32)
    clamped = np.clip(cnt, 0, cap).astype(np.int32)
    g = rng.uniform(1.0, 40.0, E).astype(np.float32)
    xb = make_acts(E, cap, K, seed=E * K)
    flat = torch.empty(offset + xb.size, dtype=torch.bfloat16, device="cuda")
    flat[offset:] = bf16_tensor(xb).reshape(-1)
    x = flat[offset:].view(E, cap, K)
    b, sf = ops.quant_act(x, dev(g), dev(cnt), 128)
    ob, valid, osf = orc.quant_act(xb, g, clamped)
    assert np.array_equal(u8(b)[valid], ob[valid]) and np.array_equal(u8(sf), osf)
    # the same rows as a gather, in reverse order and weighted
    T = E * cap
    src_tok = np.arange(T, dtype=np.int32)[::-1].copy()
    src_route = rng.permutation(T).astype(np.int32)
    w = rng.uniform(0.05, 1.0, (T, 1)).astype(np.float32)
    b2, sf2 = ops.scatter_quant_act_planned(x.reshape(T, K), dev(src_tok), dev(src_route), dev(w), dev(g), dev(cnt), cap)
    live = (np.arange(cap)[None, :] < clamped[:, None]).reshape(-1)
    dest = np.where(live, np.arange(T), T).astype(np.int64)       # T: dropped
    ob2, written, osf2 = orc.scatter_quant_act(xb.reshape(T, K), src_tok, dest, w.reshape(-1)[src_route], g, E, cap)
    assert np.array_equal(u8(b2)[written], ob2[written]) and np.array_equal(u8(sf2), osf2)


LOOKUP_CASES = [
    # E, cap, K: rows and quads - what a warp looks up at once, and where its range starts and ends inside a row
    (3, 100003, 32),       # one quad a row, more than 32 rows to a warp
    (8500, 37, 32),        # ... without prefix sums, most of them dead
    (50, 331, 288),        # three quads a row, the last with one K-block
    (5, 2, 2112),          # 17 quads a row, fewer rows than warps; K-blocks that leave the row form's lanes idle
    (40, 90, 2080),        # the same with more
    (40, 200, 2048),       # the row form, prefix in shared memory
]


@pytest.mark.parametrize("E,cap,K", LOOKUP_CASES)
def test_every_row_is_found_once(ops, E, cap, K):
    rng = np.random.default_rng(E * K)
    cnt = (rng.integers(0, cap + 1, E) * (rng.random(E) < (0.2 if E > 1000 else 0.9))).astype(np.int32)
    xb = make_acts(E, cap, K, seed=E + K)
    g = rng.uniform(1.0, 40.0, E).astype(np.float32)
    b, sf = ops.quant_act(bf16_tensor(xb), dev(g), dev(cnt), 128)
    ob, valid, osf = orc.quant_act(xb, g, cnt)
    assert np.array_equal(u8(b)[valid], ob[valid]) and np.array_equal(u8(sf), osf)
    # the gated form and the gather against the plain one, on the GPU
    x2 = bf16_tensor(np.concatenate([xb, xb[..., ::-1]], axis=-1))
    y = ops.gated_act(x2, False)
    vt = torch.from_numpy(valid).cuda()
    got, want = ops.silu_mul_quant_act(x2, dev(g), dev(cnt), 128, False), ops.quant_act(y, dev(g), dev(cnt), 128)
    assert torch.equal(got[0][vt], want[0][vt]) and torch.equal(got[1], want[1])
    src = dev(np.arange(E * cap, dtype=np.int32))
    got = ops.scatter_quant_act_planned(y.view(E * cap, K), src, src, None, dev(g), dev(cnt), cap)
    assert torch.equal(got[0][vt], want[0][vt]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("E,cap,K", [(4090, 1, 6272), (200, 130, 1056), (160, 70, 2080)])      # filled ahead (97 MiB surely dead); by the kernel
def test_planned_scatters_fill_every_dead_scale(ops, E, cap, K):
    rng = np.random.default_rng(E)
    cnt = rng.integers(0, cap + 1, E).astype(np.int32)
    T = 40
    xb = make_acts(1, T, K, seed=K)[0]
    src = rng.integers(0, T, E * cap).astype(np.int32)
    g = np.array([3.0], np.float32)
    live = np.arange(cap)[None, :] < cnt[:, None]
    dest = np.where(live.reshape(-1), np.arange(E * cap), E * cap).astype(np.int64)
    q, q_sf = ops.quant_rows(bf16_tensor(xb), dev(g))
    ob, written, osf = orc.scatter_quant_act(xb, src, dest, None, g, E, cap)
    for b, sf in (ops.scatter_quant_act_planned(bf16_tensor(xb), dev(src), dev(src), None, dev(g), dev(cnt), cap),
                  ops.scatter_fp4_planned(q, q_sf, dev(src), dev(cnt), cap)):
        assert np.array_equal(u8(sf), osf) and np.array_equal(u8(b)[written], ob[written])


@pytest.mark.parametrize("T,topk,E,cap", [(1, 1, 1, 1), (5, 7, 512, 3), (5, 7, 513, 3), (128, 8, 512, 40), (147, 7, 600, 9),
                                          (1500, 3, 512, 12), (1500, 3, 4096, 2), (341, 3, 8, 1000)])
def test_plan_around_the_ranking_tables_limit(ops, T, topk, E, cap):
    rng = np.random.default_rng(T + E)
    ids = rng.integers(-2, E + 3, (T, topk)).astype(np.int64)     # some for other ranks; repeats inside a token allowed
    counts, rd, st, sr = ops.dispatch_plan(dev(ids), 0, E, cap)
    oc, ord_, ost, osr = orc.dispatch_plan(ids, 0, E, cap)
    assert np.array_equal(u8(counts), oc) and np.array_equal(u8(rd), ord_)
    on = ost >= 0
    assert np.array_equal(u8(st)[on], ost[on]) and np.array_equal(u8(sr)[on], osr[on])


@pytest.mark.parametrize("E,M,K", [(1, 1, 32), (1, 129, 1056), (2, 128, 1024), (2, 257, 2304), (1, 300, 96), (3, 64, 1280)])
def test_compress_tile_edges(ops, E, M, K):
    rng = np.random.default_rng(M * K)
    packed, sf, _ = orc.quantize_weight(orc.prune_paired_4of8(rng.standard_normal((E, M, K)).astype(np.float32)))
    a, e, s = ops.compress(dev(packed), dev(sf), K)
    oa, oe, os_ = orc.compress(packed, sf, K)
    assert np.array_equal(u8(a), oa) and np.array_equal(u8(e), oe) and np.array_equal(u8(s), os_)


@pytest.mark.parametrize("K", [512, 3072, 3584, 8192, 1824])      # K stages 1, 6, 7, 16, 4: whole, whole, split, split, ragged
@pytest.mark.parametrize("max_n", [7, 32])
def test_narrow_gemm_with_idle_experts(ops, K, max_n):
    E, M = 70, 328
    counts = np.zeros(E, np.int32)
    counts[[0, 31, 32, 69]] = [1, max_n, 3, max_n - 1]
    rng = np.random.default_rng(K)
    w = orc.prune_paired_4of8(rng.standard_normal((4, M, K)).astype(np.float32))
    packed, sf, w_dq = orc.quantize_weight(w)
    pick = np.arange(E) % 4
    a, e, s = ops.compress(dev(packed[pick]), dev(sf[pick]), K)
    x = make_acts(E, max_n, K, K + 1)
    one = np.ones(1, np.float32)
    ob, valid, osf = orc.quant_act(x, one, counts)
    b, sfb = ops.quant_act(bf16_tensor(x), dev(one), dev(counts), M)
    al = np.linspace(0.5, 1.5, E).astype(np.float32)
    out = torch.full((E, max_n, M), -1.0, dtype=torch.bfloat16, device="cuda")
    ops.group_mm(out, a, e, s, b, sfb, dev(al), dev(counts), M, K)
    want = orc.group_mm(w_dq[pick], ob, osf, al, counts, sentinel=-1.0)
    got = out.float().cpu().numpy()
    for i in np.flatnonzero(counts):
        # bf16 rounding of the output: 2^-9 relative at most, 1.6e-3 in the norm
        assert orc.rel_frobenius(got[i, :counts[i]], want[i, :counts[i]]) <= 5e-3, i
    assert (got[~valid] == -1.0).all()


@pytest.mark.parametrize("beta,linear_beta", [(1.702, 1.0), (1.702, -1.0), (4.0, 7.0), (0.3, 0.2)])
def test_situ_against_64_bits(ops, beta, linear_beta):
    vals = (np.arange(65536, dtype=np.uint32) << 16).view(np.float32)
    ok = np.isfinite(vals) & (np.abs(vals) <= 64.0) & (np.abs(vals) >= 2.0 ** -60)
    gates = np.flatnonzero(ok).astype(np.uint16)
    gates = gates[:gates.size // 32 * 32]
    up = orc.f32_to_bf16_bits((np.random.default_rng(3).standard_normal(gates.size) * 2.0).astype(np.float32))
    x2 = np.concatenate([gates.reshape(-1, 32), up.reshape(-1, 32)], axis=1)
    y = bf16_bits(ops.gated_act(bf16_tensor(x2[None]), True, "situ", beta, linear_beta)).reshape(-1)
    g, u = (orc.bf16_bits_to_f32(v).astype(np.float64).reshape(-1) for v in (gates, up))
    want = beta * np.tanh(g / beta) / (1.0 + np.exp(-g)) * (linear_beta * np.tanh(u / linear_beta) if linear_beta > 0 else u)
    keep = np.abs(want) > 2.0 ** -100
    dist = orc.bf16_ulp_distance(y, orc.f32_to_bf16_bits(want.astype(np.float32)))[keep]
    # the float result is good to about 2^-20, half a bf16 unit is 2^-9: one value in some 1000 may round the other way
    assert dist.max() <= 1 and (dist == 0).mean() > 0.997, (dist.max(), (dist == 0).mean())


def test_gated_quantizer_passes_infinities_and_nans_like_the_chain(ops):
    rng = np.random.default_rng(5)
    x2 = orc.f32_to_bf16_bits((rng.standard_normal((2, 9, 512)) * 3).astype(np.float32))
    flat = x2.reshape(-1)
    flat[::37] = np.resize(np.array([0x7F80, 0xFF80, 0x7FC0, 0xFFC0, 0x0001, 0x8001, 0x7F7F], np.uint16), flat[::37].size)
    counts = np.array([9, 4], np.int32)
    g = dev(np.array([2.0, 30.0], np.float32))
    valid = np.arange(9)[None, :] < counts[:, None]
    for act in (("silu", 1.0, -1.0), ("situ", 1.702, 1.0)):
        y = ops.gated_act(bf16_tensor(x2), True, *act)
        got, want = ops.silu_mul_quant_act(bf16_tensor(x2), g, dev(counts), 128, True, *act), ops.quant_act(y, g, dev(counts), 128)
        assert np.array_equal(u8(got[0])[valid], u8(want[0])[valid]) and np.array_equal(u8(got[1]), u8(want[1]))
