"""Batched ALS solve (``csrc/cuda/als.cu``): W[u] = (H_u^T H_u + lambda I)^-1 H_u^T a_u."""
from __future__ import annotations

import torch

from . import _lib


def _kpad(k: int) -> int:
    for K in (32, 64, 128):
        if k <= K:
            return K
    raise ValueError("factor rank above 128 is not supported")


def als_solve(user_ptr: torch.Tensor, item_idx: torch.Tensor, rating: torch.Tensor, H: torch.Tensor,
              lam: float, seg_len: int = 4096) -> torch.Tensor:
    """``user_ptr`` (int64, n_users + 1, ascending) delimits each user's entries of ``item_idx`` (int32
    rows of H) and ``rating`` (fp32), all on one device.  Users with more than ``seg_len`` ratings are split
    over several CTAs.  Returns W [n_users, k]."""
    dev = H.device
    for name, t in (("user_ptr", user_ptr), ("item_idx", item_idx), ("rating", rating)):
        if t.device != dev:                   # their addresses go to the kernels as they are
            raise ValueError(f"{name} is on {t.device}, H on {dev}")
    H = H.contiguous().float()
    n_users, k = user_ptr.numel() - 1, H.shape[1]
    # the kernel gathers rows of H by these indices without looking at them again
    _lib.validate_ids(item_idx.contiguous(), 0, H.shape[0], "ALS ratings (item rows)")
    K = _kpad(k)
    W = torch.zeros(n_users, k, device=dev)
    nnz = item_idx.numel()
    if n_users <= 0 or nnz == 0:
        return W
    # No accumulator takes more than seg_len ratings in a row: its rounding errors grow with that.  A
    # split user's pieces are a quarter as long, so that the last ones to run are short.
    split = max(int(seg_len), 1)
    piece = max(split // 4, 256)
    # One scratch slot per split user.  nnz / split bounds them without asking the device (as long as
    # that is 4096 at most, 270 MB at rank 128), a read of the true number costs some 50 us.
    slots = nnz // split + 1
    if slots > 4096:
        slots = int(((user_ptr[1:] - user_ptr[:-1]) > split).sum().item()) + 1
    seg_cap = n_users + nnz // piece + slots
    scratch = torch.empty(slots * (K * K + K), device=dev)
    ints = torch.empty(slots + 8 + 3 * seg_cap + 4 * n_users, dtype=torch.int32, device=dev)
    slot_count, counters, seg, lists = ints.split([slots, 8, 3 * seg_cap, 4 * n_users])
    _lib.call("pcl_als_solve", user_ptr.long().contiguous(), item_idx.int().contiguous(),
              rating.float().contiguous(), H, W, scratch, slot_count, counters, seg, lists, n_users, split, piece,
              seg_cap, k, float(lam), _lib.stream_ptr())
    return W
