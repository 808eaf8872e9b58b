// Kernels of the device SVD (alternating least squares + Cholesky-QR; reference:
// alg/recommendation/svd/svd.hpp:137-181 for the products A.H and A^T.W that it forms with
// Eigen on every worker, 221-231 for the Cholesky-QR):
//
//   spmm_csr      out[r, :]  = sum_j A[r, c_j] * H[c_j, :]      (K <= 128)
//   spmm_csr_t    out[c, :] += A[r, c] * W[r, :]                (vector reductions, fp32)
//   chol_factor   G = L L^T for a small K x K Gram matrix; writes R = L^T and T = L^-T so that
//                 Q = M T is orthonormal and M = Q R, and G^-1 = T T^T.  One CTA, fp64 in
//                 shared memory.  A pivot below the tolerance marks the matrix rank deficient in
//                 `info` (index of the pivot + 1) and the caller falls back to an
//                 eigen-decomposition.
#include "common.cuh"

namespace {

// Work is cut by entries, not by rows: a group of G lanes (the smallest power of two with 16 bytes
// of a K-wide row per lane) owns SP_L consecutive entries whatever rows they belong to, so a row with a
// million entries is spread over the chip and a row with two costs two.  (A warp per row took 13.7 ms
// on 400 k rows x 16 M Zipf(1.1) entries, K = 32, of which one warp's chain over the hottest row was all
// but half a millisecond, and used 8 of its 32 lanes; SPMM_MEAS.)  What is left is bound by the
// gathers of 4 K bytes per entry out of L2: four are in flight per group before the first is used.
// A segment that holds a whole row stores it; the pieces of a cut row are added with vector
// reductions into `out`, which the launcher clears.
// TRANS: out[c, :] += v * W[r, :] instead (a reduction per entry; W's row stays in registers).
constexpr int SP_ROWS = 1024;   // row ends of a block kept in shared memory up to this many rows

// largest r in [0, n_rows) with row_ptr[r] <= e, for row_ptr[0] <= e < row_ptr[n_rows]; one warp,
// 32 probes at a time
__device__ __forceinline__ long long row_of_entry(const long long* row_ptr, long long n_rows, long long e,
                                                  int lane) {
  long long lo = 0, hi = n_rows;            // row_ptr[lo] <= e < row_ptr[hi]
  while (hi - lo > 1) {
    const long long step = (hi - lo + 32) / 33 > 0 ? (hi - lo + 32) / 33 : 1;
    const long long probe = lo + (lane + 1) * step;
    const bool le = probe < hi && __ldg(row_ptr + probe) <= e;
    const int cnt = __popc(__ballot_sync(0xffffffffu, le));
    const long long nhi = lo + (cnt + 1) * step;
    lo += cnt * step;
    hi = nhi < hi ? nhi : hi;
  }
  return lo;
}

template <int G, bool TRANS>
__global__ void __launch_bounds__(256) spmm_kernel(const long long* __restrict__ row_ptr,
                                                   const int* __restrict__ cols,
                                                   const float* __restrict__ vals, long long n_rows,
                                                   long long n_ent, int L, const float* __restrict__ X,
                                                   int K, float* __restrict__ out) {
  constexpr int GPB = 256 / G;
  __shared__ int s_end[SP_ROWS];            // ends of the block's rows relative to its first entry
  __shared__ long long s_row[2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  long long e0 = (long long)blockIdx.x * GPB * L, e1 = e0 + (long long)GPB * L;
  const long long base = e0;
  const long long first = __ldg(row_ptr), last = __ldg(row_ptr + n_rows);
  if (e0 < first) e0 = first;
  if (e1 > last) e1 = last;
  if (e1 > n_ent) e1 = n_ent;
  if (e0 >= e1) return;                     // uniform over the block
  if (warp < 2) {
    const long long r = row_of_entry(row_ptr, n_rows, warp == 0 ? e0 : e1 - 1, lane);
    if (lane == 0) s_row[warp] = r;
  }
  __syncthreads();
  const long long r0 = s_row[0];
  const long long nrows = s_row[1] - r0 + 1;
  const bool cached = nrows <= SP_ROWS;
  auto rel = [&](long long q) -> int {      // q relative to base, saturated to the block
    const long long d = q - base;
    return d > 0x3fffffff ? 0x3fffffff : (d < -1 ? -1 : (int)d);
  };
  if (cached)
    for (int i = threadIdx.x; i < (int)nrows; i += 256) s_end[i] = rel(__ldg(row_ptr + r0 + i + 1));
  __syncthreads();
  auto row_end = [&](long long i) -> int { return cached ? s_end[i] : rel(__ldg(row_ptr + r0 + i + 1)); };
  const int g = threadIdx.x / G, gl = threadIdx.x % G;
  int gs = g * L, ge = gs + L;
  if (gs < (int)(e0 - base)) gs = (int)(e0 - base);
  if (ge > (int)(e1 - base)) ge = (int)(e1 - base);
  if (gs >= ge) return;
  const bool on = 4 * gl < K;
  // row of the group's first entry
  long long i = 0;
  {
    long long lo = 0, hi = nrows - 1;       // smallest i with row_end(i) > gs
    while (lo < hi) {
      const long long mid = (lo + hi) >> 1;
      if (row_end(mid) > gs) hi = mid; else lo = mid + 1;
    }
    i = lo;
  }
  int end = row_end(i);
  // whether the current row starts before this segment
  bool cut = i > 0 ? row_end(i - 1) < gs : rel(__ldg(row_ptr + r0)) < gs;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (TRANS && on) acc = __ldg(reinterpret_cast<const float4*>(X + (r0 + i) * K + 4 * gl));
  auto flush = [&](bool cut_here) {
    float* o = out + (r0 + i) * K + 4 * gl;
    if (on) {
      if (cut_here) pcl_red_add4(o, acc);
      else *reinterpret_cast<float4*>(o) = acc;
    }
  };
  constexpr int U = 4;
  const bool vec = ((reinterpret_cast<uintptr_t>(cols) | reinterpret_cast<uintptr_t>(vals)) & 15) == 0;
  for (int p0 = gs & ~(U - 1); p0 < ge; p0 += U) {
    int c[U];
    float v[U];
    const long long q = base + p0;
    if (vec && q + U <= n_ent) {
      const int4 c4 = __ldg(reinterpret_cast<const int4*>(cols + q));
      c[0] = c4.x; c[1] = c4.y; c[2] = c4.z; c[3] = c4.w;
      if (vals) {
        const float4 v4 = __ldg(reinterpret_cast<const float4*>(vals + q));
        v[0] = v4.x; v[1] = v4.y; v[2] = v4.z; v[3] = v4.w;
      } else {
        v[0] = v[1] = v[2] = v[3] = 1.f;
      }
    } else {
#pragma unroll
      for (int j = 0; j < U; ++j) {
        const bool in = q + j < n_ent;
        c[j] = in ? __ldg(cols + q + j) : 0;
        v[j] = in && vals ? __ldg(vals + q + j) : 1.f;
      }
    }
    float4 h[U];
    if constexpr (!TRANS) {
#pragma unroll
      for (int j = 0; j < U; ++j)
        h[j] = (on && p0 + j >= gs && p0 + j < ge) ? __ldg(reinterpret_cast<const float4*>(X + (long long)c[j] * K + 4 * gl))
                                                   : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int p = p0 + j;
      if (p < gs || p >= ge) continue;
      if (p >= end) {
        if constexpr (!TRANS) flush(cut);
        do end = row_end(++i); while (p >= end);
        cut = false;
        acc = make_float4(0.f, 0.f, 0.f, 0.f);
        if (TRANS && on) acc = __ldg(reinterpret_cast<const float4*>(X + (r0 + i) * K + 4 * gl));
      }
      if constexpr (TRANS) {
        if (on && v[j] != 0.f)
          pcl_red_add4(out + (long long)c[j] * K + 4 * gl,
                       make_float4(v[j] * acc.x, v[j] * acc.y, v[j] * acc.z, v[j] * acc.w));
      } else {
        acc.x = fmaf(v[j], h[j].x, acc.x); acc.y = fmaf(v[j], h[j].y, acc.y);
        acc.z = fmaf(v[j], h[j].z, acc.z); acc.w = fmaf(v[j], h[j].w, acc.w);
      }
    }
  }
  if constexpr (!TRANS) flush(cut || end > ge);
}

template <bool TRANS>
int launch_spmm(const long long* row_ptr, const int* cols, const float* vals, long long n_rows,
                long long n_ent, const float* X, int K, float* out, cudaStream_t stream) {
  int G = 1;
  while (4 * G < K) G *= 2;
  // entries per group: 128, fewer while the chip's groups (2048 threads on each of 148 SMs) would
  // not all get a segment
  int L = 128;
  while (L > 16 && n_ent / L < 148LL * 2048 / G) L /= 2;
  const long long blocks = (n_ent + (256 / G) * (long long)L - 1) / ((256 / G) * (long long)L);
  if (blocks > 0x7fffffffLL) return (int)cudaErrorInvalidValue;
#define PCL_SPMM(GG)                                                                                     \
  case GG:                                                                                               \
    spmm_kernel<GG, TRANS><<<(int)blocks, 256, 0, stream>>>(row_ptr, cols, vals, n_rows, n_ent, L, X, K, out); \
    break;
  switch (G) {
    PCL_SPMM(1) PCL_SPMM(2) PCL_SPMM(4) PCL_SPMM(8) PCL_SPMM(16) PCL_SPMM(32)
  }
#undef PCL_SPMM
  return pcl_last_error();
}

// One CTA.  Shared memory: L (K x K doubles) and X = L^-1 (K x K doubles).
__global__ void __launch_bounds__(256) chol_factor_kernel(const float* __restrict__ G, int K,
                                                          float* __restrict__ T, float* __restrict__ R,
                                                          double rel_tol, int* __restrict__ info) {
  extern __shared__ double sd[];
  double* L = sd;
  double* X = sd + (size_t)K * K;
  __shared__ double s_diag, s_max;
  __shared__ int s_bad;
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int e = tid; e < K * K; e += nt) {
    const int i = e / K, j = e % K;
    L[e] = 0.5 * ((double)G[i * K + j] + (double)G[j * K + i]);   // symmetrise
    X[e] = 0.0;
  }
  if (tid == 0) { s_bad = 0; s_max = 0.0; }
  __syncthreads();
  if (tid == 0) {
    double m = 0.0;
    for (int i = 0; i < K; ++i) m = fmax(m, fabs(L[i * K + i]));
    s_max = m;
  }
  __syncthreads();
  // right-looking Cholesky on the lower triangle
  for (int j = 0; j < K; ++j) {
    if (tid == 0) {
      const double d = L[j * K + j];
      if (!(d > rel_tol * s_max) && s_bad == 0) s_bad = j + 1;
      s_diag = d > 0.0 ? sqrt(d) : 1.0;
    }
    __syncthreads();
    if (s_bad) break;
    const double dj = s_diag;
    for (int i = j + tid; i < K; i += nt) L[i * K + j] = (i == j) ? dj : L[i * K + j] / dj;
    __syncthreads();
    // trailing update: L[i][k] -= L[i][j] * L[k][j] for j < k <= i
    const int rem = K - j - 1;
    for (int e = tid; e < rem * rem; e += nt) {
      const int i = j + 1 + e / rem, k = j + 1 + e % rem;
      if (k <= i) L[i * K + k] -= L[i * K + j] * L[k * K + j];
    }
    __syncthreads();
  }
  if (s_bad) {
    if (tid == 0) *info = s_bad;
    return;
  }
  // X = L^-1 by forward substitution, one column per thread
  for (int c = tid; c < K; c += nt) {
    for (int i = c; i < K; ++i) {
      double s = (i == c) ? 1.0 : 0.0;
      for (int k = c; k < i; ++k) s -= L[i * K + k] * X[k * K + c];
      X[i * K + c] = s / L[i * K + i];
    }
  }
  __syncthreads();
  for (int e = tid; e < K * K; e += nt) {
    const int i = e / K, j = e % K;
    R[e] = (j >= i) ? (float)L[j * K + i] : 0.f;     // R = L^T (upper)
    T[e] = (j >= i) ? (float)X[j * K + i] : 0.f;     // T = (L^-1)^T (upper)
  }
  if (tid == 0) *info = 0;
}

}  // namespace

// CSR of n_rows rows whose entries lie in cols / vals [0, n_ent) (vals null: ones).  X and out are
// 16-byte aligned with K <= 128 a multiple of 4.
PCL_API int pcl_spmm_csr(const long long* row_ptr, const int* cols, const float* vals, long long n_rows,
                         long long n_ent, const float* H, int K, float* out, cudaStream_t stream) {
  if (n_rows <= 0) return 0;
  if (K <= 0 || K > 128 || (K & 3)) return (int)cudaErrorInvalidValue;
  cudaError_t e = cudaMemsetAsync(out, 0, (size_t)n_rows * K * sizeof(float), stream);
  if (e != cudaSuccess) return (int)e;
  if (n_ent <= 0) return 0;
  return launch_spmm<false>(row_ptr, cols, vals, n_rows, n_ent, H, K, out, stream);
}

PCL_API int pcl_spmm_csr_t(const long long* row_ptr, const int* cols, const float* vals, long long n_rows,
                           long long n_ent, const float* W, int K, float* out, cudaStream_t stream) {
  if (n_rows <= 0 || n_ent <= 0) return 0;
  if (K <= 0 || K > 128 || (K & 3)) return (int)cudaErrorInvalidValue;
  return launch_spmm<true>(row_ptr, cols, vals, n_rows, n_ent, W, K, out, stream);
}

PCL_API int pcl_chol_factor(const float* G, int K, float* T, float* R, double rel_tol, int* info,
                            cudaStream_t stream) {
  if (K <= 0 || K > 112) return (int)cudaErrorInvalidValue;   // 2 K^2 doubles must fit in 227 KB
  const size_t smem = 2 * (size_t)K * K * sizeof(double);
  cudaError_t e = cudaFuncSetAttribute(chol_factor_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return (int)e;
  chol_factor_kernel<<<1, 256, smem, stream>>>(G, K, T, R, rel_tol, info);
  return pcl_last_error();
}
