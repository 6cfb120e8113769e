"""The work a program that uses this package has it do, as cases that can be timed and compared.

Every case goes through the public entry points (torch.ops.paired_nvfp4.*, paired_nvfp4_kernels.ep).  Kinds:

  layer     one MoE layer of the serving loop for a batch of routed tokens: dispatch_plan ->
            scatter_quant_act_planned -> gate_up (fused with activation and requantization, or group_mm followed by
            silu_mul_quant_act) -> group_mm (down) -> moe_finalize; eager, or replayed from a CUDA graph that holds it
  batched   the same expert FFN on activations that are already batched by expert: quant_act -> gate_up -> down
  linear    one grouped linear layer: quant_act -> group_mm
  ep        paired_nvfp4_kernels.ep.ExpertParallelFFN.forward on one rank that holds every expert
  load      compress of one layer's gate_up weights, as a model loader calls it

Tactics: "tuned" is the tile choice that bench.py makes (512-K stages on 64-token tiles up to 64 rows per expert,
256-token tiles on CTA pairs above), "suggested" what paired_nvfp4_kernels.suggest_tactic returns, for programs that
do not autotune.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.abspath("grouped-sparse-gemm_b200"))
import paired_nvfp4_kernels as pnk  # noqa: E402
from paired_nvfp4_kernels import ep, reference  # noqa: E402

ops = torch.ops.paired_nvfp4

WSTD = 0.02            # standard deviation of the synthetic weights
BANK_ROWS = 2048       # distinct quantized weight rows; the rows of a weight are drawn from them
# fused gate_up variant with the tile of a group_mm variant (ids as listed by the package)
FUSED_OF = {"sparse_1sm_128x64_k512": "fused_2sm_256x64_k512", "sparse_2sm_256x256": "fused_2sm_256x256",
            "sparse_1sm_128x64": "fused_1sm_128x64", "sparse_2sm_256x128": "fused_2sm_256x128"}


def _layer(name, tokens, experts, hidden, inter, topk, cap, **more):
    case = dict(name=name, kind="layer", tokens=tokens, experts=experts, experts_total=experts, first=0, hidden=hidden,
                inter=inter, topk=topk, cap=cap, fused=True, activation="silu", interleaved=True, weight_on="output",
                routing="normal", tactic="tuned", graph=False)
    case.update(more)
    return case


def listed():
    return [
        # one user's decode step: a single token, eight small experts, launch latency only
        _layer("one_token", 1, 128, 2048, 768, 8, 16),
        # decode of a batch on eight large experts whose rows arrive batched by expert: the weights' bytes
        dict(name="decode_batched", kind="batched", experts=8, hidden=4096, inter=14336, cap=16, fused=True,
             activation="silu", interleaved=True, tactic="tuned"),
        # decode on one rank's 32 of 256 experts, the whole layer replayed from a CUDA graph as a server does
        _layer("decode_graph", 128, 32, 7168, 2048, 8, 32, experts_total=256, first=96, graph=True),
        # a larger decode batch on large experts, tile variant as suggested: between the decode and prefill kernels
        _layer("decode_wide", 100, 8, 4096, 14336, 2, 100, tactic="suggested"),
        # a small grouped linear layer with ragged row counts, default tile variant
        dict(name="linear_small", kind="linear", experts=8, features=2048, hidden=1024, cap=256, tactic="suggested"),
        # a short prompt (odd token count) on many small experts, tile variant as suggested
        _layer("short_prompt", 777, 128, 2048, 768, 8, 128, tactic="suggested"),
        # prefill with sizes that are no multiple of the kernels' tiles, unfused, plain [gate | up] layout, router
        # weights applied to the input
        _layer("odd_prefill", 3001, 32, 2880, 2880, 4, 768, fused=False, interleaved=False, weight_on="input"),
        # prefill of 16384 tokens on 128 small experts
        _layer("prefill", 16384, 128, 2048, 768, 8, 2048),
        # the prefill share of one of eight ranks: 32 experts, 2048 rows each
        _layer("prefill_shard", 8192, 32, 7168, 2048, 8, 4096),
        # skewed routing (Zipf), SiTU activation, unfused, interleaved layout
        _layer("skewed", 8192, 128, 3072, 3072, 4, 4096, routing="zipf", activation="situ", fused=False),
        # expert-parallel layer on one rank with all 256 experts
        dict(name="expert_parallel", kind="ep", tokens=8192, experts=256, hidden=7168, inter=2048, topk=8, cap=1024,
             tactic="tuned"),
        # loading a model: the compressor on one layer's gate_up weights
        dict(name="load", kind="load", experts=8, features=28672, hidden=4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cap_for(tokens, topk, experts_total):
    if tokens <= 64:
        return max(16, -(-tokens // 16) * 16)
    mean = tokens * topk / experts_total
    return min(tokens, max(64, -(-int(2 * mean) // 128) * 128))


def draw(rng):
    kind = rng.choice(["layer"] * 11 + ["batched"] * 2 + ["linear"] * 3 + ["ep"] * 2 + ["load"] * 2)
    tactic = rng.choice(["tuned", "tuned", "suggested"])
    if kind == "load":
        k = 32 * _log_int(rng, 16, 224)
        m = 64 * _log_int(rng, 8, 448)
        e = max(1, min(64, int(4e8 / (m * k / 2))))
        return dict(kind=kind, experts=rng.randint(1, e), features=m, hidden=k)
    if kind == "linear":
        e, m, k = _log_int(rng, 1, 64), 8 * _log_int(rng, 32, 1024), 32 * _log_int(rng, 8, 224)
        cap = _log_int(rng, 1, max(16, min(2048, int(3e12 / (2.0 * e * m * k)))))
        return dict(kind=kind, experts=e, features=m, hidden=k, cap=cap, tactic=tactic)
    activation = rng.choice(["silu", "silu", "silu", "situ"])
    if kind == "batched":
        e, h, i = rng.choice([(8, 4096, 14336), (16, 4096, 6400), (32, 7168, 2048), (64, 2048, 1408)])
        cap = _log_int(rng, 1, 256)
        return dict(kind=kind, experts=e, hidden=h, inter=i, cap=cap, fused=rng.random() < 0.75, activation=activation,
                    interleaved=True, tactic=tactic)
    # models: experts, hidden, intermediate, top-k
    e, h, i, topk = rng.choice([(8, 4096, 14336, 2), (128, 2048, 768, 8), (256, 7168, 2048, 8), (128, 3072, 3072, 4),
                                (32, 2880, 2880, 4), (64, 2048, 1408, 6), (16, 5120, 8192, 1),
                                (rng.choice([12, 40, 96]), 32 * rng.randint(32, 160), 64 * rng.randint(8, 48), rng.randint(1, 8))])
    most = min(16384, int(4e12 / (6.0 * topk * h * i)))
    tokens = _log_int(rng, 1, most)
    if kind == "ep":
        return dict(kind=kind, tokens=tokens, experts=e, hidden=h, inter=i, topk=topk,
                    cap=_cap_for(tokens, topk, e), tactic=tactic)
    local, first = e, 0
    if e > 32 and rng.random() < 0.4:            # one rank's share of the experts
        local = e // rng.choice([2, 4, 8])
        first = local * rng.randrange(e // local)
    fused = rng.random() < 0.7
    return _layer(None, tokens, local, h, i, topk, _cap_for(tokens, topk, e), experts_total=e, first=first, fused=fused,
                  activation=activation, interleaved=True if fused else rng.random() < 0.5,
                  weight_on=rng.choice(["output", "output", "input"]), routing=rng.choice(["normal", "normal", "zipf"]),
                  tactic=tactic, graph=rng.random() < 0.25) | {"name": "drawn"}


# ------------------------------------------------------------------------------------------------ inputs

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _packed_weights(experts, features, k, g):
    """Gaussian weights, pruned and quantized as the checkpoint format wants them (codes, block scales)."""
    bank = torch.randn((1, BANK_ROWS, k), generator=g, device="cuda") * WSTD
    codes, scales, _ = reference.quantize_weight(reference.prune_paired_4of8(bank))
    rows = torch.randint(BANK_ROWS, (experts * features,), generator=g, device="cuda")
    return (codes[0].index_select(0, rows).view(experts, features, k // 2),
            scales[0].index_select(0, rows).view(experts, features, k // 32))


def _compressed(experts, features, k, g):
    codes, scales = _packed_weights(experts, features, k, g)
    return ops.compress(codes, scales, k)


def _weights(case, g):
    """w13 ([gate; up], rows interleaved where the layout says so: the rows are independent draws, so the layout is
    a matter of how the outputs are read) and w2."""
    e, h, i = case["experts"], case["hidden"], case["inter"]
    return _compressed(e, 2 * i, h, g), _compressed(e, h, i, g)


def _scales(case, x):
    """Global scales of the two quantizers and the matching alphas: amax of the input; a static estimate between the
    GEMMs, as a calibrated checkpoint carries."""
    e = case["experts"]
    g1 = (6.0 * 448.0 / x.abs().max().float()).expand(e).contiguous()
    sigma = WSTD * math.sqrt(case["hidden"])
    amax2 = 1.702 if case.get("activation") == "situ" else max(1.0, (5.0 * sigma) ** 2)
    g2 = torch.full((e,), 6.0 * 448.0 / amax2, device="cuda")
    return g1, 1.0 / g1, g2, 1.0 / g2


def _tactic(case):
    """(group_mm config, cluster_m), (fused config, cluster_m)"""
    names, fused_names = pnk.group_mm_configs(), list(ops.group_mm_swiglu_configs())
    if case["tactic"] == "suggested":
        cid, cm, _ = pnk.suggest_tactic(case["cap"])
    else:
        cid = names.index("sparse_1sm_128x64_k512" if case["cap"] <= 64 else "sparse_2sm_256x256")
        cm = 2 if "_2sm_" in names[cid] else 1
    fid = fused_names.index(FUSED_OF[names[cid]])
    return (cid, cm), (fid, 2 if "_2sm_" in fused_names[fid] else 1)


def _activation(case):
    return (case["activation"],) + ((1.702, 1.0) if case["activation"] == "situ" else (1.0, -1.0))


def _routing(case, g):
    t, e, topk = case["tokens"], case.get("experts_total", case["experts"]), case["topk"]
    logits = torch.randn((t, e), generator=g, device="cuda")
    if case.get("routing") == "zipf":
        rank = torch.randperm(e, generator=g, device="cuda").float() + 1
        logits += torch.log(rank ** -1.2 / (rank ** -1.2).sum())
    top = logits.topk(topk, dim=-1)
    return top.indices.contiguous(), torch.softmax(top.values, -1).contiguous()


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    s = dict(case=case, kind=kind)
    if kind == "load":
        s["codes"], s["scales"] = _packed_weights(case["experts"], case["features"], case["hidden"], g)
        return s
    bf16 = dict(dtype=torch.bfloat16, device="cuda")
    e, h, cap = case["experts"], case["hidden"], case["cap"]
    s["tactic"], s["fused_tactic"] = _tactic(case)
    if kind in ("batched", "linear"):
        x = torch.randn((e, cap, h), generator=g, device="cuda").to(torch.bfloat16)
        s["counts"] = torch.randint(1, cap + 1, (e,), generator=g, device="cuda", dtype=torch.int32)
    else:
        x = torch.randn((case["tokens"], h), generator=g, device="cuda").to(torch.bfloat16)
        s["ids"], s["router_w"] = _routing(case, g)
        s["final"] = torch.zeros((case["tokens"], h), **bf16)
    s["x"] = x
    s["g1"], s["al1"], s["g2"], s["al2"] = _scales(case, x)
    if kind == "linear":
        s["w"] = _compressed(e, case["features"], h, g)
        s["out"] = torch.zeros((e, cap, case["features"]), **bf16)
        return s
    s["w13"], s["w2"] = _weights(case, g)
    if kind == "ep":
        t, topk = case["tokens"], case["topk"]
        s["ffn"] = ep.ExpertParallelFFN(s["w13"], s["w2"], h, case["inter"], cap, s["al1"], s["al2"], s["g1"][:1].contiguous(),
                                        s["g2"], ep.slab_rows(t, topk, 1), fused_config=s["fused_tactic"][0],
                                        config_id=s["tactic"][0], cluster_m=s["tactic"][1],
                                        fused_cluster_m=s["fused_tactic"][1], world=1, rank=0)
        return s
    s["act"] = _activation(case)
    if not case["fused"]:
        s["mid"] = torch.zeros((e, cap, 2 * case["inter"]), **bf16)
    s["out"] = torch.zeros((e, cap, h), **bf16)
    if case.get("graph"):
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _moe_layer(s)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            s["held"] = _moe_layer(s)
        s["graph"] = graph
    return s


# ------------------------------------------------------------------------------------------------ one pass

def _expert_ffn(s, b1, sf1, counts):
    """gate_up, activation, down on quantized rows batched by expert; the result is in s["out"]."""
    case = s["case"]
    h, i = case["hidden"], case["inter"]
    (cid, cm), (fid, fcm) = s["tactic"], s["fused_tactic"]
    if case["fused"]:
        b2, sf2 = ops.group_mm_swiglu_quant(*s["w13"], b1, sf1, s["al1"], counts, s["g2"], 2 * i, h, fid, fcm, 1, *s["act"])
    else:
        ops.group_mm(s["mid"], *s["w13"], b1, sf1, s["al1"], counts, 2 * i, h, cid, cm, 1)
        b2, sf2 = ops.silu_mul_quant_act(s["mid"], s["g2"], counts, h, case["interleaved"], *s["act"])
    ops.group_mm(s["out"], *s["w2"], b2, sf2, s["al2"], counts, h, i, cid, cm, 1)


def _moe_layer(s):
    case = s["case"]
    e, cap = case["experts"], case["cap"]
    on_input = case["weight_on"] == "input"
    counts, route_dest, src_tok, src_route = ops.dispatch_plan(s["ids"], case["first"], e, cap)
    b1, sf1 = ops.scatter_quant_act_planned(s["x"], src_tok, src_route, s["router_w"] if on_input else None, s["g1"], counts, cap)
    _expert_ffn(s, b1, sf1, counts)
    ops.moe_finalize(s["final"], s["out"], route_dest, None if on_input else s["router_w"])
    return s["final"], counts


def run(s):
    kind = s["kind"]
    if kind == "layer":
        if "graph" in s:
            s["graph"].replay()
            return s["held"]
        return _moe_layer(s)
    if kind == "batched":
        b1, sf1 = ops.quant_act(s["x"], s["g1"], s["counts"], 2 * s["case"]["inter"])
        _expert_ffn(s, b1, sf1, s["counts"])
        return s["out"]
    if kind == "linear":
        m, k = s["case"]["features"], s["case"]["hidden"]
        b, sf = ops.quant_act(s["x"], s["g1"], s["counts"], m)
        ops.group_mm(s["out"], *s["w"], b, sf, s["al1"], s["counts"], m, k, s["tactic"][0], s["tactic"][1], 1)
        return s["out"]
    if kind == "ep":
        return s["ffn"].forward(s["x"], s["ids"], s["router_w"], s["final"])
    return ops.compress(s["codes"], s["scales"], s["case"]["hidden"])


# ------------------------------------------------------------------------------------------------ what a pass needs

def _up(a, b):
    return -(-a // b) * b


def _weight_bytes(m, k):
    """codes, metadata and scales of one expert's [m, k] weight"""
    return m * k / 4 + _up(m, 128) * _up(k, 256) / 16 + _up(m, 128) * _up(-(-k // 32), 4)


def _quantized(rows, k):
    return rows * (k / 2 + k / 32)


def work(case):
    """Every call's inputs read once and its outputs written once; rows and active experts are expectations over the
    routing (uniform, where it is not skewed)."""
    kind, e, h = case["kind"], case["experts"], case["hidden"]
    if kind == "load":
        m = case["features"]
        return {"bytes": e * (m * h / 2 + m * h / 32 + _weight_bytes(m, h)), "flops": 0}
    if kind == "linear":
        m, rows = case["features"], e * (case["cap"] + 1) / 2
        return {"bytes": rows * 2 * h + 2 * _quantized(rows, h) + e * _weight_bytes(m, h) + rows * 2 * m, "flops": 2.0 * rows * m * h}
    i = case["inter"]
    if kind == "batched":
        rows, active = e * (case["cap"] + 1) / 2, e
        around = rows * 2 * h + _quantized(rows, h)
    else:
        t, topk, total = case["tokens"], case["topk"], case.get("experts_total", e)
        rows = min(t * topk * e / total, e * case["cap"])
        active = e * (1 - (1 - topk / total) ** t)
        around = t * topk * 12 + rows * 8 + t * 2 * h + _quantized(rows, h)          # plan, quantize
        around += rows * 2 * h + t * 2 * h + t * topk * 4                            # combine
        if kind == "ep":                                                             # quantize once, pack, plan again, place
            around += 2 * _quantized(t, h) + 2 * _quantized(rows, h) + t * topk * 12 + rows * 8
    fused = case.get("fused", True)
    mid = _quantized(rows, i) if fused else 2 * rows * 4 * i + _quantized(rows, i)
    ffn = active * (_weight_bytes(2 * i, h) + _weight_bytes(h, i)) + _quantized(rows, h) + mid + _quantized(rows, i) + rows * 2 * h
    return {"bytes": around + ffn, "flops": 6.0 * rows * h * i}


def tolerance(case):
    # compressed weights are bytes; everything else ends in bf16, after a second 4-bit quantization whose codes may
    # round the other way where the first GEMM's bf16 result differs in its last bit
    return "exact" if case["kind"] == "load" else {"rel": 1e-2}
