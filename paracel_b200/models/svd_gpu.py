"""Truncated SVD on GPUs (device path of alg/recommendation/svd/svd.hpp:40-310 and of the
complete serial version tool/svd_serial.cpp:40-190).

``SvdGpu`` is a ``paralg`` subclass on the device backend.  The sparse matrix A is
row-partitioned over the ranks (CSR in HBM), H (N x K) is replicated, W (local rows x K) is
local.  Stage 1 repeats ``W = A H (H^T H)^-1``, ``H = A^T W (W^T W)^-1``; the K x K Gram matrix
``W^T W`` and the N x K product ``A^T W`` are summed over the ranks THROUGH the parameter
tables, as the reference does with its ``WtW`` / ``AtW_<k>`` keys (svd.hpp:137-181): each rank
writes its part into ``paracel_delta_buffer(key)`` and a collective ``paracel_bupdate`` with the
``svd_updater`` (add) handler reduces them into the owners' shards, ``paracel_read`` gathers the
sum.  Stage 2 is the Cholesky-QR of W and H (``M^T M = R^T R``, ``Q = M R^-1``) and the SVD of the
K x K matrix ``R_W R_H^T`` (on the host, svd.hpp:294-298), ``U = Q_W U_r``, ``V = Q_H V_r``.

Kernels: CSR products ``A.H`` / ``A^T.W`` (the second on a transposed copy of A made by ``load``, or by
scattered additions where the matrix is too large for a copy),
products of a tall matrix with a K x K one and the small Cholesky factor (csrc/cuda/svd.cu), and the
Gram matrix (``pcl_gram``)."""
from __future__ import annotations

import os

import torch

from ..ops.misc import gram
from ..ops.svd import chol_factor, host_rand, rows_times, spmm_csr, spmm_csr_t
from ..paralg import paralg


# Pivots and eigenvalues of a Gram matrix summed in fp32 are rounding noise below about this much of the
# largest, and a direction scaled by one over its noise spoils the others.  With cuts of 1e-10 and 1e-12 a
# singular value of an exact rank-12 matrix was off by more than 0.2 % in one solve of eight and those of a
# rank-60 one by a factor; cuts from 2^-25 to 2^-22 are good to 1e-6 on both.  Larger ones lose
# singular values of a thousandth of the largest.
_GRAM_NOISE = 2.0 ** -24


def _orth_fallback(G: torch.Tensor):
    """(T, R) from the eigen-decomposition of a semi-definite Gram matrix restricted to its
    numerical range: Q = M T is orthonormal and M = Q R."""
    lam, V = torch.linalg.eigh(G.double().cpu())
    keep = lam > _GRAM_NOISE * lam.max()
    lam, V = lam[keep], V[:, keep]
    T = (V / lam.sqrt()[None, :]).float()
    R = (V * lam.sqrt()[None, :]).T.float()
    return T.to(G.device), R.to(G.device)


def _transpose_fits(entries: int, n_cols: int, free_bytes: int) -> bool:
    """Whether ``load`` makes a transposed copy of the matrix.  torch.sort takes up to 2^31 - 1 elements,
    and the copy, 8 bytes an entry once made, passes through keys, 8-byte positions and their sort
    buffers: 64 bytes an entry and 24 a column at most, which may take half of what is free."""
    return entries < 1 << 31 and 64 * entries + 24 * n_cols <= free_bytes // 2


class SvdGpu(paralg):
    def __init__(self, n_cols: int, k: int = 2, iters: int = 20, oversample: int = 10, seed: int = 0,
                 group=None, device=None, comm=None, hosts_dct_str=None, output: str = "",
                 update_function: str = "svd_updater"):
        super().__init__(hosts_dct_str, comm, output, backend="gpu", device=device, group=group)
        self.world, self.rank, self.group = self.get_worker_size(), self.get_worker_id(), group
        self.N, self.k, self.iters, self.seed = int(n_cols), int(k), int(iters), seed
        K = min(self.k + int(oversample), self.N)
        self.K = min((K + 3) // 4 * 4, 112)
        self.update_function = update_function
        self.paracel_dense_table("WtW", self.K * self.K, handler=update_function)
        self.paracel_dense_table("AtW", self.N * self.K, handler=update_function)

    def load(self, row_ptr: torch.Tensor, cols: torch.Tensor, vals: torch.Tensor):
        """This rank's rows of A as CSR (int64 row_ptr, int32 global column ids, fp32 values).  Also makes a
        transposed copy where `_transpose_fits`; larger matrices do without."""
        from ..ops import _lib
        dev = self.device
        self.row_ptr = row_ptr.to(dev, torch.int64).contiguous()
        self.cols = cols.to(dev, torch.int32).contiguous()
        self.vals = vals.to(dev, torch.float32).contiguous()
        _lib.validate_ids(self.cols, 0, self.N, "SVD input (column ids)")
        self.m = self.row_ptr.numel() - 1
        first, last = (int(self.row_ptr[0].item()), int(self.row_ptr[-1].item())) if self.m > 0 else (0, 0)
        self.t_ptr = self.t_rows = self.t_vals = None
        free = 1 << 29                    # small matrices do without asking, which takes 0.2 ms
        if not _transpose_fits(last - first, self.N, free):
            free = torch.cuda.mem_get_info(dev)[0] + torch.cuda.memory_reserved(dev) - torch.cuda.memory_allocated(dev)
        if not _transpose_fits(last - first, self.N, free):
            return
        # A^T in the same form: its products then add up in registers.  Scattering an entry at a time
        # into A^T W queues up at the popular columns: 1 ms a product on 6.5 M Zipf(1.1) entries,
        # K = 32, against 0.14 ms for A H.
        c, order = torch.sort(self.cols[first:last], stable=True)
        row_of = torch.repeat_interleave(torch.arange(self.m, device=dev, dtype=torch.int32),
                                         self.row_ptr[1:] - self.row_ptr[:-1], output_size=last - first)
        self.t_rows, self.t_vals = row_of[order], self.vals[first:last][order]
        self.t_ptr = torch.searchsorted(c, torch.arange(self.N + 1, device=dev, dtype=torch.int32))

    def _times_transposed(self, W: torch.Tensor, out: torch.Tensor) -> None:
        """``out = A^T W`` for this rank's rows."""
        if self.t_ptr is not None:
            spmm_csr(self.t_ptr, self.t_rows, self.t_vals, W, out)
        else:
            spmm_csr_t(self.row_ptr, self.cols, self.vals, W, out.zero_())

    def _reduce(self, key: str, buf: torch.Tensor, cols: int) -> torch.Tensor:
        """Sum over the ranks of what each wrote into ``buf``, the delta buffer of the table ``key``:
        owners start from zero, a collective bupdate adds every rank's part, a read gathers the result."""
        self.paracel_local_shard(key).zero_()
        self.paracel_bupdate(key, buf, "", self.update_function, collective=True)
        return self.paracel_read(key).view(-1, cols).clone()

    def _sum_gram(self, W: torch.Tensor) -> torch.Tensor:
        """``W^T W`` over all ranks."""
        buf = self.paracel_delta_buffer("WtW").zero_()
        if self.m:
            gram(W, buf.view(self.K, self.K))
        return self._reduce("WtW", buf, self.K)

    def _times_inverse(self, M: torch.Tensor, G: torch.Tensor) -> torch.Tensor:
        """``M @ pinv(G)`` for a K x K Gram matrix: ``(M T) T^T`` with the Cholesky factor, or
        the pseudo-inverse when G is rank deficient (the oversampled factors can be)."""
        if M.shape[0] == 0:
            return M
        T, _, info = chol_factor(G, rel_tol=_GRAM_NOISE)
        if info != 0:
            Tf, _ = _orth_fallback(G)
            return (M @ Tf) @ Tf.T
        return rows_times(M, T, twice=True)

    def _orth(self, G: torch.Tensor):
        T, R, info = chol_factor(G, rel_tol=_GRAM_NOISE)
        if info != 0:
            return _orth_fallback(G)
        return T, R

    def solve(self):
        dev, K, N = self.device, self.K, self.N
        H = host_rand((N, K), self.seed, dev, 2.0, -1.0)          # same H on every rank
        A = (self.row_ptr, self.cols, self.vals)
        for _ in range(self.iters):
            W = self._times_inverse(spmm_csr(*A, H), gram(H))
            WtW = self._sum_gram(W)
            buf = self.paracel_delta_buffer("AtW")
            self._times_transposed(W, buf.view(N, K))
            AtW = self._reduce("AtW", buf, K)
            H = self._times_inverse(AtW, WtW)
        W = self._times_inverse(spmm_csr(*A, H), gram(H))
        Tw, Rw = self._orth(self._sum_gram(W))
        Th, Rh = self._orth(gram(H))
        def times(M, T):
            if M.shape[0] == 0 or T.shape[0] != T.shape[1]:
                return M @ T
            return rows_times(M, T)
        Qw, Qh = times(W, Tw), times(H, Th)
        Ur, S, Vrt = torch.linalg.svd((Rw @ Rh.T).double().cpu())      # small K x K problem on the host
        kk = min(self.k, S.numel())
        self.sigma = S[:kk].clone()
        self.U = (Qw @ Ur.float().to(dev))[:, :kk].contiguous()
        self.V = (Qh @ Vrt.T.float().to(dev))[:, :kk].contiguous()
        self.paracel_sync()
        self.paracel_check()

    def dump_result(self, outdir: str = "", row_names=None, col_names=None):
        """SIGMA_0 and V_0 from worker 0, U_<rank> from every worker (tool/svd_serial.cpp:140-153)."""
        from ..utils.dump import dump_dict_vector, dump_vector
        outdir = outdir or self.output
        os.makedirs(outdir, exist_ok=True)
        if self.rank == 0:
            dump_vector(self.sigma.tolist(), os.path.join(outdir, "SIGMA_0"))
            cn = col_names if col_names is not None else list(range(self.N))
            dump_dict_vector({cn[j]: row for j, row in enumerate(self.V.cpu().tolist())},
                             os.path.join(outdir, "V_0"))
        rn = row_names if row_names is not None else list(range(self.m))
        dump_dict_vector({rn[j]: row for j, row in enumerate(self.U.cpu().tolist())},
                         os.path.join(outdir, f"U_{self.rank}"))
        self.paracel_sync()

    def free(self):
        self.close()
