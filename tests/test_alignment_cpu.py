"""Pointers that a kernel's vector loads and stores cannot take are refused on the host, before anything is launched: an
operand may be a contiguous piece of a larger buffer at any element offset."""
import pytest

A = 0x100000           # stands for an aligned device address; nothing reads it
INVALID = 1            # PNV_ERR_INVALID_ARGUMENT


@pytest.fixture(scope="module")
def cabi():
    from paired_nvfp4_kernels import _cabi
    return _cabi


# entry point, arguments with the pointer under test as a letter, {letter: offsets that are refused}
CALLS = [
    ("pnv_quant_act", ("x", A, 0, A, 2, 16, 64, "b", "s", 0, None), dict(x=(2, 8), b=(1, 4), s=(1, 2))),
    ("pnv_silu_mul_quant_act", ("x", A, 0, A, 2, 16, 64, 1, 0, 1.0, -1.0, "b", "s", 0, None), dict(x=(2, 8), b=(1, 4), s=(1, 2))),
    ("pnv_scatter_quant_act", ("x", A, A, None, A, 0, 5, 64, 2, 16, "b", "s", 0, None), dict(x=(2, 8), b=(4, 8), s=(1, 2))),
    ("pnv_scatter_quant_act_planned", ("x", A, A, None, A, 0, A, 64, 2, 16, "b", "s", 0, None), dict(x=(2, 8), b=(4, 8), s=(1, 2))),
    ("pnv_scatter_fp4_planned", ("x", A, A, A, 128, 2, 16, "b", A, 0, None), dict(x=(1, 8), b=(1, 8))),
    ("pnv_quant_rows", ("x", A, 5, 128, "b", "s", 0, None), dict(x=(2, 8), b=(1, 8), s=(1, 2))),
    ("pnv_gated_act", ("x", 5, 64, 0, 0, 1.0, -1.0, "b", None), dict(x=(2, 8), b=(2, 8))),
    ("pnv_moe_finalize", ("b", "x", A, None, 5, 2, 64, None), dict(x=(2, 8), b=(2, 8))),
    ("pnv_compress", ("x", A, 2, 16, 64, "b", "m", "s", None), dict(x=(1, 2), b=(4, 8), m=(1, 2), s=(4, 8))),
]


@pytest.mark.parametrize("name,args,refused", CALLS, ids=[c[0] for c in CALLS])
def test_misaligned_pointers_are_refused(cabi, name, args, refused):
    for letter, offsets in refused.items():
        for off in offsets:
            rc = getattr(cabi.lib, name)(*[(A + off if a == letter else A) if isinstance(a, str) else a for a in args])
            msg = cabi.lib.pnv_last_error().decode()
            assert rc == INVALID and "aligned" in msg, (letter, off, rc, msg)
