"""No-GPU checks of the operator layer and of its build."""
import pytest
import torch

INTEGER_OR_NO_RESULTS = [
    "compress", "quant_act", "silu_mul_quant_act", "scatter_quant_act", "dispatch_plan", "scatter_quant_act_planned",
    "quant_rows", "scatter_fp4_planned", "moe_finalize", "pack_wire_rows", "scatter_fp4_wire", "group_mm", "group_mm_rows",
    "zero_rows", "group_mm_rows_parts", "zero_rows_parts", "pack_wire_rows_parts", "group_mm_swiglu_quant"]
FLOAT_RESULTS = ["gather_rows", "gated_act"]


@pytest.fixture(scope="module")
def pnk():
    import paired_nvfp4_kernels
    return paired_nvfp4_kernels


def test_only_ops_without_float_results_pass_autograd_by(pnk):
    """torch's autograd fallback marks floating-point results as having no backward; nothing else it does could be seen
    on integer results or written arguments."""
    def has_autograd_kernel(op):
        return torch._C._dispatch_has_kernel_for_dispatch_key(f"paired_nvfp4::{op}", "AutogradCUDA")

    assert [op for op in FLOAT_RESULTS if has_autograd_kernel(op)] == []
    assert [op for op in INTEGER_OR_NO_RESULTS if not has_autograd_kernel(op)] == []
