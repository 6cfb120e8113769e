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
