"""What surrounds torch.ops.paired_nvfp4.* on the Python side.  The operators themselves (argument validation, output
allocation, stream lookup) are C++, csrc/torch_ops.cpp; importing this module loads and registers them.
"""
import ctypes
import os

import torch

from . import _cabi

_lib = _cabi.lib
SF_BLOCK = 32          # dense K elements per scale
TORCH_LIB_PATH = os.path.join(os.path.dirname(_cabi.LIB_PATH), "libpaired_nvfp4_torch.so")


def _load():
    if not os.path.exists(TORCH_LIB_PATH):
        raise ImportError(f"{TORCH_LIB_PATH} is missing: build it with `python grouped-sparse-gemm_b200/build.py`. "
                          "There is no CPU or PyTorch fallback for these ops.")
    try:
        torch.ops.load_library(TORCH_LIB_PATH)
        lib = ctypes.CDLL(TORCH_LIB_PATH)
    except OSError as exc:  # pragma: no cover
        raise ImportError(f"could not load {TORCH_LIB_PATH}: {exc} (it loads into the torch it was built for: after a change of "
                          "torch run `python grouped-sparse-gemm_b200/build.py`)") from exc
    lib.pnv_torch_set_sm_margin.argtypes = [ctypes.c_int]
    lib.pnv_torch_set_sm_margin.restype = None
    return lib


_torch_lib = _load()


def _check(cond, msg):
    if not cond:
        raise RuntimeError(msg)


def set_sm_margin(n):
    """Leave `n` SMs out of every persistent launch (the kernels size their grids from the SM count passed
    in), so that a collective running on another stream finds SMs to run on.  0 restores full-width launches."""
    _torch_lib.pnv_torch_set_sm_margin(max(0, int(n)))


def wire_row_bytes(k):
    """Bytes of one wire row of the expert-parallel dispatch for hidden size k."""
    return int(_lib.pnv_wire_row_bytes(int(k)))


def wire_expert_ids(wire):
    """The [rows, 1] int32 view of the expert ids inside wire rows (input of dispatch_plan on the receiver)."""
    _check(wire.dim() == 2 and wire.dtype == torch.uint8 and wire.is_contiguous() and wire.size(1) % 16 == 0,
           "wire must be contiguous uint8 [rows, wire_row_bytes(K)]")
    rb = wire.size(1)
    return wire.view(torch.int32)[:, rb // 4 - 4: rb // 4 - 3]


def set_silu_table(enabled):
    """Testing aid: evaluate SiLU in the library's short form (default) or by the expression itself."""
    _cabi.check(_lib.pnv_set_silu_table(1 if enabled else 0))


def group_mm_device_status():
    """Status word of the bounded waits inside group_mm (0 = all completed); synchronises."""
    v = ctypes.c_int()
    _cabi.check(_lib.pnv_group_mm_device_status(ctypes.byref(v)))
    return v.value


def __getattr__(name):
    """The operators under this module's name too: ops.quant_act is torch.ops.paired_nvfp4.quant_act."""
    if name.startswith("__"):
        raise AttributeError(name)
    return getattr(torch.ops.paired_nvfp4, name)
