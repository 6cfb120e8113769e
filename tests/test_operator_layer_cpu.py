"""No-GPU checks of the operator layer and of its build."""
import importlib.util
import os

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


@pytest.mark.skipif(torch.cuda.is_available(), reason="the call would be launched; its pointers stand for nothing")
def test_quantizers_take_more_than_two_to_the_31_rows(pnk):
    """E * max_n of 2^31 and beyond fits this GPU's memory at K = 32 (64 + 16 + 4 bytes a row): refused neither by the
    argument checks nor by a 32-bit row number.  (Without a device the launch itself fails, with another code.)"""
    from paired_nvfp4_kernels import _cabi
    p = 0x100000
    rc = _cabi.lib.pnv_quant_act(p, p, 0, p, 2, 1 << 30, 32, p, p, 148, None)
    assert rc == 2, _cabi.lib.pnv_last_error()
    rc = _cabi.lib.pnv_quant_act(p, p, 0, p, 4, (1 << 30) - 1, 32, p, p, 148, None)
    assert rc == 1 and b"2^32" in _cabi.lib.pnv_last_error()


def test_names_of_the_ops_module(pnk):
    """Everything a program could take from paired_nvfp4_kernels.ops: the operators under their own names, the helpers, the
    block size of the scales."""
    from paired_nvfp4_kernels import ops
    assert ops.SF_BLOCK == 32
    for name in INTEGER_OR_NO_RESULTS + FLOAT_RESULTS + [
            "group_mm_configs", "group_mm_swiglu_configs", "set_sm_margin", "wire_row_bytes", "wire_expert_ids",
            "set_silu_table", "group_mm_device_status"]:
        assert callable(getattr(ops, name)), name
    with pytest.raises(AttributeError):
        ops.no_such_operator


def test_the_operator_library_is_rebuilt_for_another_torch(pnk, monkeypatch):
    """C++ against torch's headers does not load into another torch, whatever the files' times say."""
    path = os.path.join(os.path.dirname(os.path.dirname(pnk.__file__)), "build.py")
    spec = importlib.util.spec_from_file_location("pnv_build", path)
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    assert torch.__version__ in build.torch_build_id() and torch.version.git_version in build.torch_build_id()
    assert build.torch_ops_up_to_date()
    monkeypatch.setattr(build, "torch_build_id", lambda: "torch-build:0.0:none;")
    assert not build.torch_ops_up_to_date()
