"""C entry points of the quantizers on destinations that are less than 16-byte aligned: an operand may be a piece of a
larger buffer.  (Sources and destinations a kernel cannot take are refused on the host: test_alignment_cpu.py.)"""
import numpy as np
import pytest
import torch

from helpers import bf16_tensor, dev, make_acts

pytestmark = pytest.mark.gpu

E, CAP = 3, 70
COUNTS = np.array([70, 0, 33], np.int32)


@pytest.fixture(scope="module")
def lib():
    from paired_nvfp4_kernels import _cabi
    return _cabi


def at_offset(n, offset):
    """n bytes that start `offset` bytes into an allocation, and the guard bytes around them."""
    flat = torch.full((offset + n + 64,), 0xA5, dtype=torch.uint8, device="cuda")
    return flat, flat[offset:offset + n]


def untouched(flat, offset, n):
    return bool((flat[:offset] == 0xA5).all()) and bool((flat[offset + n:] == 0xA5).all())


def same_rows(got, want, k):
    live = torch.arange(CAP, device="cuda")[None, :] < dev(COUNTS)[:, None]
    return torch.equal(got.view(E, CAP, k // 2)[live], want.view(E, CAP, k // 2)[live])


@pytest.mark.parametrize("K", [96, 2048])
@pytest.mark.parametrize("b_off,sf_off", [(8, 0), (8, 4), (0, 4)])
def test_quant_act_and_silu_mul(lib, K, b_off, sf_off):
    ops = torch.ops.paired_nvfp4
    cnt, g = dev(COUNTS), dev(np.array([3.0, 5.0, 7.0], np.float32))
    stream = torch.cuda.current_stream().cuda_stream
    x, x2 = bf16_tensor(make_acts(E, CAP, K, K)), bf16_tensor(make_acts(E, CAP, 2 * K, K + 1))
    n_b, n_sf = E * CAP * K // 2, lib.sf_numel(CAP, K, E)
    for want, call in (
            (ops.quant_act(x, g, cnt, 128),
             lambda b, s: lib.lib.pnv_quant_act(x.data_ptr(), g.data_ptr(), 1, cnt.data_ptr(), E, CAP, K, b, s, 0, stream)),
            (ops.silu_mul_quant_act(x2, g, cnt, 128, True),
             lambda b, s: lib.lib.pnv_silu_mul_quant_act(x2.data_ptr(), g.data_ptr(), 1, cnt.data_ptr(), E, CAP, K, 1, 0, 1.0, -1.0,
                                                         b, s, 0, stream))):
        (fb, b), (fs, s) = at_offset(n_b, b_off), at_offset(n_sf, sf_off)
        lib.check(call(b.data_ptr(), s.data_ptr()))
        assert same_rows(b, want[0], K) and torch.equal(s, want[1])
        assert untouched(fb, b_off, n_b) and untouched(fs, sf_off, n_sf)


@pytest.mark.parametrize("K,sf_off", [(96, 4), (96, 1), (2048, 4), (2048, 2)])
def test_planned_scatters(lib, K, sf_off):
    ops = torch.ops.paired_nvfp4
    T, stream = 50, torch.cuda.current_stream().cuda_stream
    x = bf16_tensor(make_acts(1, T, K, K))[0]
    cnt, g = dev(COUNTS), torch.full((1,), 3.0, device="cuda")
    src = dev((np.arange(E * CAP) * 7 % T).astype(np.int32))
    n_b, n_sf = E * CAP * K // 2, lib.sf_numel(CAP, K, E)
    q, q_sf = ops.quant_rows(x, g)
    want = ops.scatter_fp4_planned(q, q_sf, src, cnt, CAP)
    calls = [lambda b, s: lib.lib.pnv_scatter_fp4_planned(q.data_ptr(), q_sf.data_ptr(), src.data_ptr(), cnt.data_ptr(), K, E, CAP,
                                                          b, s, 0, stream)]
    if sf_off == 4:        # (this one always writes words)
        calls.append(lambda b, s: lib.lib.pnv_scatter_quant_act_planned(x.data_ptr(), src.data_ptr(), src.data_ptr(), None,
                                                                        g.data_ptr(), 0, cnt.data_ptr(), K, E, CAP, b, s, 0, stream))
    for call in calls:
        (_, b), (fs, s) = at_offset(n_b, 0), at_offset(n_sf, sf_off)
        lib.check(call(b.data_ptr(), s.data_ptr()))
        assert same_rows(b, want[0], K) and torch.equal(s, want[1])
        assert untouched(fs, sf_off, n_sf)


@pytest.mark.parametrize("interleaved", [False, True])
def test_gated_act_on_a_source_that_is_16_byte_aligned(interleaved):
    ops = torch.ops.paired_nvfp4
    x2 = bf16_tensor(make_acts(1, 37, 2 * 96, 3))[0]
    flat = torch.empty(8 + x2.numel(), dtype=torch.bfloat16, device="cuda")
    flat[8:] = x2.view(-1)
    for act in (("silu", 1.0, -1.0), ("situ", 1.702, 1.0)):
        assert torch.equal(ops.gated_act(flat[8:].view(37, 192), interleaved, *act), ops.gated_act(x2, interleaved, *act))
