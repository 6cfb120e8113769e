"""What the operator layer keeps, allocates and tells autograd."""
import warnings

import numpy as np
import pytest
import torch

from helpers import dev

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    import paired_nvfp4_kernels  # noqa: F401
    return torch.ops.paired_nvfp4


@pytest.mark.parametrize("op", ["gated_act", "gather_rows"])
def test_float_results_say_that_they_have_no_backward(ops, op):
    w = torch.randn((3, 64), dtype=torch.bfloat16, device="cuda", requires_grad=True)
    call = {"gated_act": lambda t: ops.gated_act(t, True),
            "gather_rows": lambda t: ops.gather_rows(t, dev(np.array([2, -1, 0, 0], np.int32)))}[op]
    y = call(w * 2)
    assert y.requires_grad and y.grad_fn is not None
    with warnings.catch_warnings(record=True) as seen:
        warnings.simplefilter("always")
        y.float().sum().backward()
    assert any("autograd kernel was not registered" in str(m.message) for m in seen)
    with torch.no_grad():
        assert torch.equal(call(w * 2), y) and not call(w * 2).requires_grad
    q, _ = ops.quant_act(w.view(1, 3, 64), torch.ones(1, device="cuda"), dev(np.array([3], np.int32)), 128)
    assert not q.requires_grad


def test_uninitialised_rows_are_filled_where_torch_fills_them(ops):
    """Under torch.use_deterministic_algorithms the bytes that no kernel writes are torch's fill value, as for torch.empty."""
    counts = dev(np.array([2, 0, 5], np.int32))
    x = torch.randn((3, 5, 64), device="cuda").to(torch.bfloat16)
    ids = dev(np.array([[0, 2], [0, 2], [2, 2], [2, 2]], np.int64))
    before = torch.are_deterministic_algorithms_enabled(), torch.is_deterministic_algorithms_warn_only_enabled()
    torch.use_deterministic_algorithms(True)
    try:
        b, _ = ops.quant_act(x, torch.ones(1, device="cuda"), counts, 128)
        plan_counts, _, src_tok, src_route = ops.dispatch_plan(ids, 0, 3, 8)
    finally:
        torch.use_deterministic_algorithms(before[0], warn_only=before[1])
    assert bool((b[0, 2:] == 255).all()) and bool((b[1] == 255).all())
    dead = torch.arange(8, device="cuda")[None, :] >= plan_counts[:, None]
    assert plan_counts.tolist() == [2, 0, 6]
    for t in (src_tok, src_route):
        assert bool((t.view(3, 8)[dead] == torch.iinfo(torch.int32).max).all())


# ---- split-K workspaces ------------------------------------------------------------------------------------------

K_SPLIT = 3584         # seven K stages of 512


class SplitProblem:
    """A narrow GEMM over many experts of which four are active.  The first `e` experts of every operand are operands of a
    problem of their own, with another number of arrival counters and the same four experts' results."""
    M, MAX_N, E = 256, 16, 1088

    def __init__(self, ops, seed):
        from helpers import make_acts, make_weights, bf16_tensor
        self.ops = ops
        packed, sf, _ = make_weights(4, self.M, K_SPLIT, seed, 0.05)
        pick = np.arange(self.E) % 4
        self.a, self.meta, self.sfa = ops.compress(dev(packed).index_select(0, dev(pick)), dev(sf).index_select(0, dev(pick)), K_SPLIT)
        x = bf16_tensor(make_acts(4, self.MAX_N, K_SPLIT, seed + 1)).index_select(0, dev(pick))
        counts = np.zeros(self.E, np.int32)
        counts[:4] = [16, 1, 7, 16]
        self.counts = dev(counts)
        self.one = torch.ones(self.E, device="cuda")
        self.b, self.sfb = ops.quant_act(x, self.one, self.counts, self.M)

    def run(self, e, out=None):
        if out is None:
            out = torch.zeros((e, self.MAX_N, self.M), dtype=torch.bfloat16, device="cuda")
        self.ops.group_mm(out, self.a[:e], self.meta[:e], self.sfa, self.b[:e], self.sfb, self.one[:e], self.counts[:e], self.M,
                          K_SPLIT, 7, 1, 1)
        return out


@pytest.fixture(scope="module")
def split_problem(ops):
    from helpers import splits_k
    p = SplitProblem(ops, 5)
    for e in (32, p.E):
        assert splits_k(e, p.M, K_SPLIT, p.MAX_N, [16, 1, 7, 16])
    return p


def test_a_captured_workspace_goes_with_its_call(split_problem):
    """Every live block of a graph's private pool belongs to somebody outside the library once the capture is over."""
    p = split_problem
    want = p.run(32).clone()
    out = torch.zeros_like(want)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(3):
            p.run(32, out)
    pool = tuple(graph.pool())
    live = [b["size"] for s in torch.cuda.memory_snapshot() if tuple(s["segment_pool_id"]) == pool
            for b in s["blocks"] if b["state"] == "active_allocated"]
    assert live == []
    for _ in range(3):                        # replays between eager calls of this and of another size
        out.zero_()
        graph.replay()
        assert torch.equal(out, want)
        assert torch.equal(p.run(32), want) and torch.equal(p.run(1088)[:4], want[:4])


def test_captures_leave_the_eager_workspaces_alone(split_problem):
    p = split_problem
    want = p.run(32).clone()
    outs = [torch.zeros((32 * (i + 2), p.MAX_N, p.M), dtype=torch.bfloat16, device="cuda") for i in range(33)]
    graphs = []
    for out in outs:
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1]):
            p.run(out.size(0), out)
    out = torch.zeros_like(want)
    before = torch.cuda.memory_stats()["allocation.all.allocated"]
    p.run(32, out)
    assert torch.cuda.memory_stats()["allocation.all.allocated"] == before, "the call had to allocate its workspace again"
    for g, o in zip(graphs, outs):
        g.replay()
        assert torch.equal(o[:4], want[:4])
    assert torch.equal(out, want)


def test_more_sizes_than_workspaces_are_kept(split_problem):
    """34 problems with 34 numbers of arrival counters in turn, twice: the oldest workspaces have gone back by the time
    their size returns."""
    p = split_problem
    want = p.run(32).clone()
    for _ in range(2):
        for e in range(32, p.E + 1, 32):
            got = p.run(e)
            assert torch.equal(got[:4], want[:4]) and not got[4:].any(), e
    assert torch.equal(p.run(32), want)
    from paired_nvfp4_kernels import ops as pyops
    assert pyops.group_mm_device_status() == 0


def test_workspaces_of_two_streams_and_sizes(split_problem):
    """Two streams, two sizes each, interleaved: no launch sees another's counters or partial sums."""
    p = split_problem
    want = p.run(32).clone()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    outs = []
    for i in range(6):
        for s in streams:
            with torch.cuda.stream(s):
                outs += [p.run(32), p.run(128 + 32 * (i & 1))]
    torch.cuda.synchronize()
    assert all(torch.equal(o[:4], want[:4]) for o in outs)
