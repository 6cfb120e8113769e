"""Seeded input builders shared by the GPU parity tests (numpy on the host, torch for device I/O)."""
import numpy as np
import torch

from oracle import paired_nvfp4_oracle as orc


def bf16_tensor(bits, device="cuda"):
    """uint16 bf16 bit patterns -> torch.bfloat16 tensor on `device`."""
    return torch.from_numpy(np.ascontiguousarray(bits).view(np.int16)).view(torch.bfloat16).to(device)


def bf16_bits(t):
    """torch.bfloat16 tensor -> uint16 bit patterns (numpy, host)."""
    return t.detach().contiguous().view(torch.int16).cpu().numpy().view(np.uint16)


def u8(t):
    return t.detach().contiguous().cpu().numpy()


def dev(a, dtype=None):
    t = torch.from_numpy(np.ascontiguousarray(a))
    if dtype is not None:
        t = t.to(dtype)
    return t.cuda()


def make_weights(E, M, K, seed, scale=1.0):
    """Seeded N(0, scale) weights -> pruned paired-4:8 -> NVFP4.  Returns (packed, sf, dequant)."""
    rng = np.random.default_rng(seed)
    w = (rng.standard_normal((E, M, K)) * scale).astype(np.float32)
    return orc.quantize_weight(orc.prune_paired_4of8(w))


def make_acts(E, max_n, K, seed, scale=1.0):
    rng = np.random.default_rng(seed)
    return orc.f32_to_bf16_bits((rng.standard_normal((E, max_n, K)) * scale).astype(np.float32))


def splits_k(E, M, K, max_n, counts, sms=148):
    """Does group_mm cut the K stages of this problem across CTAs?  The kernel's own rule, with its constants read from the
    sources, so that a test of the split path notices when a changed rule no longer takes it there."""
    import os
    import re
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    header = open(os.path.join(root, "include", "paired_nvfp4_b200.h")).read()
    source = open(os.path.join(root, "grouped-sparse-gemm_b200", "csrc", "group_mm.cu")).read()
    min_k = int(re.search(r"#define PNV_SPLIT_MIN_K (\d+)", header).group(1))
    saves = int(re.search(r"constexpr int kSplitSaves = (\d+);", source).group(1))
    assert "2 * n_tiles < 3 * grid" in source and "ksn >= q + 1 + kSplitSaves" in source
    m_tiles, stages = -(-M // 128), -(-K // 512)
    grid = min(E * m_tiles * stages, sms)
    tiles = sum(1 for c in counts if c > 0) * m_tiles
    return max_n <= 32 and K >= min_k and 2 * tiles < 3 * grid and stages >= tiles * stages // grid + 1 + saves
