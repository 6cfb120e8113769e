"""paired_nvfp4_kernels for B200 (sm_100a): paired-4:8 sparse NVFP4 grouped MoE GEMM ops.

Importing this package loads ``libpaired_nvfp4_b200.so`` (hand-written sm_100a CUDA behind a C ABI)
and ``libpaired_nvfp4_torch.so``, which registers ``torch.ops.paired_nvfp4.*`` with the reference project's
operator schemas (csrc/ops.cu:739-773), so code written against the reference's package runs unchanged.  The helper
surface of the reference's ``paired_nvfp4_kernels/__init__.py`` (tactic enumeration, the gate/up
interleave permutation, availability probes) is provided under the same names.

There is no CPU or eager-PyTorch fallback: without the compiled libraries the import fails.
"""
import torch

from . import _cabi, ops

__version__ = "0.1.0"

__all__ = [
    "DEFAULT_TACTIC",
    "all_tactics",
    "fused_swiglu_tactics",
    "interleave_gate_up_rows",
    "built_archs",
    "group_mm_configs",
    "is_available",
    "loaded_arch",
    "suggest_tactic",
    "valid_clusters",
]

_LOADED_SM = 100

# (config_id, cluster_m, cluster_n): also the schema defaults of torch.ops.paired_nvfp4.group_mm (csrc/torch_ops.cpp)
DEFAULT_TACTIC = (0, 2, 1)
_CLUSTER_DIMS = (1, 2, 4)


def _current_sm():
    if not torch.cuda.is_available():
        return None
    major, minor = torch.cuda.get_device_capability()
    return major * 10 + minor


def loaded_arch():
    """SM number the loaded library was built for (100)."""
    return _LOADED_SM


def built_archs():
    """SM numbers with compiled kernels in this installation."""
    return [_LOADED_SM]


def is_available():
    """Can the ops run here?  Needs a CUDA device of the architecture the library was built for (the
    operators themselves are registered at import, or the import would have failed)."""
    return _current_sm() == _LOADED_SM and all(
        hasattr(torch.ops.paired_nvfp4, op) for op in ("compress", "quant_act", "group_mm"))


def group_mm_configs():
    """Names of the tile variants, indexed by config_id."""
    return list(torch.ops.paired_nvfp4.group_mm_configs())


def _needs_cta_pair(config_name):
    """Variant names read <kind>_<1sm|2sm>_<rows>x<tokens>[_k512]; "2sm" variants run on pairs of CTAs."""
    fields = config_name.split("_")
    return len(fields) > 1 and fields[1] == "2sm"


def valid_clusters(config_name, max_product=16):
    """(cluster_m, cluster_n) pairs the op accepts for one tile variant: both from {1, 2, 4}, product at most
    max_product, and an even cluster_m where the variant runs on CTA pairs."""
    pair = _needs_cta_pair(config_name)
    return [(cm, cn) for cm in _CLUSTER_DIMS for cn in _CLUSTER_DIMS
            if cm * cn <= max_product and not (pair and cm % 2 == 1)]


def all_tactics(max_cluster_product=16):
    """Every candidate (config_id, cluster_m, cluster_n); the op re-validates each one."""
    return [(cid, cm, cn) for cid, name in enumerate(group_mm_configs())
            for cm, cn in valid_clusters(name, max_cluster_product)]


def interleave_gate_up_rows(n, device=None):
    """Row order of W13 ([gate; up], 2n rows) for a GEMM whose epilogue pairs gate and up values:
    64-row blocks holding gate rows 32b..32b+31 followed by up rows n+32b..n+32b+31.  Apply to the
    dense packed weight and its block scales before compress().  n must be a multiple of 64."""
    if n % 64:
        raise ValueError(f"intermediate size must be a multiple of 64, got {n}")
    gate = torch.arange(n, device=device).view(n // 32, 1, 32)
    return torch.cat([gate, gate + n], dim=1).reshape(-1)


def fused_swiglu_tactics(max_cluster_product=16):
    """Candidate (config_id, cluster_m, cluster_n) for group_mm_swiglu_quant; empty if the fused op is absent."""
    configs = getattr(torch.ops.paired_nvfp4, "group_mm_swiglu_configs", None)
    if configs is None:
        return []
    tactics = []
    for cid, name in enumerate(configs()):
        tactics.extend((cid, cm, cn) for cm, cn in valid_clusters(name, max_cluster_product))
    return tactics


def suggest_tactic(max_n):
    """A reasonable group_mm tactic for a per-expert token capacity of max_n, without autotuning:
    64-column tiles when max_n fits one, the 128-column default otherwise."""
    names = group_mm_configs()
    if max_n <= 64:
        return (names.index("sparse_1sm_128x64"), 1, 1)
    return DEFAULT_TACTIC
