"""Wrappers of the device SVD kernels (``csrc/cuda/svd.cu``): CSR x dense products with a
skinny right-hand side, tall matrices times small square ones, the host generator's stream on the
device and the Cholesky factor of a small Gram matrix."""
from __future__ import annotations

from typing import Optional, Tuple

import torch

from . import _lib


def spmm_csr(row_ptr: torch.Tensor, cols: torch.Tensor, vals: Optional[torch.Tensor], H: torch.Tensor,
             out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``A @ H`` for CSR ``A`` (int64 row_ptr, int32 cols, fp32 vals or None for ones) and dense
    ``H [N, K]`` with ``K <= 128`` a multiple of 4."""
    _lib.check_cuda(H, torch.float32, "H")
    n, K = row_ptr.numel() - 1, H.shape[1]
    if out is None:
        out = torch.empty(n, K, device=H.device)
    _lib.call("pcl_spmm_csr", row_ptr, cols, vals, n, cols.numel(), H, K, out, _lib.stream_ptr())
    return out


def spmm_csr_t(row_ptr: torch.Tensor, cols: torch.Tensor, vals: Optional[torch.Tensor], W: torch.Tensor,
               out: torch.Tensor) -> torch.Tensor:
    """``out += A.T @ W`` for CSR ``A`` with ``n`` rows and dense ``W [n, K]``; ``out [N, K]``."""
    _lib.check_cuda(W, torch.float32, "W")
    _lib.check_cuda(out, torch.float32, "out")
    n, K = row_ptr.numel() - 1, W.shape[1]
    _lib.call("pcl_spmm_csr_t", row_ptr, cols, vals, n, cols.numel(), W, K, out, _lib.stream_ptr())
    return out


def rows_times(M: torch.Tensor, P: torch.Tensor, twice: bool = False) -> torch.Tensor:
    """``M @ P`` or, with ``twice``, ``(M @ P) @ P.T`` for ``M [n, K]`` and ``P [K, K]``, K <= 112 a
    multiple of 4."""
    _lib.check_cuda(M, torch.float32, "M")
    _lib.check_cuda(P, torch.float32, "P")
    K = M.shape[1]
    if P.shape != (K, K) or K % 4 or K > 112 or (M.data_ptr() & 15):
        raise ValueError("P must be K x K for the K <= 112 columns of an aligned M, K a multiple of 4")
    out = torch.empty_like(M)
    _lib.call("pcl_rows_times", M, M.shape[0], K, P, int(twice), out, _lib.stream_ptr())
    return out


def host_rand(shape, seed: int, device, scale: float = 1.0, shift: float = 0.0) -> torch.Tensor:
    """``torch.rand(shape, generator=g) * scale + shift`` for a fresh CPU generator ``g`` with
    ``manual_seed(seed)``, made on the device (number for number where the scaled values are exact,
    as they are for 2 and -1)."""
    if type(seed) is not int or not 0 <= seed < 1 << 32:       # plain seeds need no generator, 10 us
        g = torch.Generator()
        g.manual_seed(seed)                    # refuses what the generator refuses, maps negative seeds
        seed = g.initial_seed()
    if torch.device(device).type != "cuda":
        raise ValueError("the numbers are made on a CUDA device")
    out = torch.empty(shape, device=device, dtype=torch.float32)
    _lib.call("pcl_mt19937_uniform", out, out.numel(), seed & 0xffffffff, float(scale), float(shift),
              _lib.stream_ptr())
    return out


def chol_factor(G: torch.Tensor, rel_tol: float = 1e-10) -> Tuple[torch.Tensor, torch.Tensor, int]:
    """For a symmetric positive definite ``G [K, K]`` (K <= 112): ``(T, R, info)`` with
    ``G = R^T R``, ``T = R^-1`` (so ``M T`` is orthonormal when ``G = M^T M`` and
    ``G^-1 = T T^T``).  ``info`` > 0 is the (1-based) pivot at which the factorisation met a
    value below ``rel_tol`` times the largest diagonal entry; T and R are then undefined."""
    _lib.check_cuda(G, torch.float32, "G")
    K = G.shape[0]
    T = torch.empty(K, K, device=G.device)
    R = torch.empty(K, K, device=G.device)
    info = torch.zeros(1, dtype=torch.int32, device=G.device)
    _lib.call("pcl_chol_factor", G, K, T, R, float(rel_tol), info, _lib.stream_ptr())
    return T, R, int(info.item())
