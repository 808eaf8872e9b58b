// Kernels of the device SVD (alternating least squares + Cholesky-QR; reference:
// alg/recommendation/svd/svd.hpp:137-181 for the products A.H and A^T.W that it forms with
// Eigen on every worker, 221-231 for the Cholesky-QR):
//
//   spmm_csr      out[r, :]  = sum_j A[r, c_j] * H[c_j, :]      (K <= 128)
//   spmm_csr_t    out[c, :] += A[r, c] * W[r, :]                (vector reductions, fp32)
//   rows_times    out = M P, or (M P) P^T, for tall M and a small square P (K <= 112)
//   mt19937       the start matrix: U(0, 1) of the host generator of the same seed
//   chol_factor   G = L L^T for a small K x K Gram matrix; writes R = L^T and T = L^-T so that
//                 Q = M T is orthonormal and M = Q R, and G^-1 = T T^T.  One CTA, fp64 in
//                 shared memory.  A pivot below the tolerance marks the matrix rank deficient in
//                 `info` (index of the pivot + 1) and the caller falls back to an
//                 eigen-decomposition.
#include "common.cuh"

namespace {

// Work is cut by entries, not by rows: a group of G lanes (the smallest power of two with 16 bytes
// of a K-wide row per lane) owns L consecutive entries whatever rows they belong to, so a row with a
// million entries is spread over the chip and a row with two costs two.  (A warp per row took 13.7 ms
// on 400 k rows x 16 M Zipf(1.1) entries, K = 32, of which one warp's chain over the hottest row was all
// but half a millisecond, and used 8 of its 32 lanes.)  What is left is bound by the
// gathers of 4 K bytes per entry out of L2: four are in flight per group before the first is used.
// Rows of even length, against a warp per row: 500 k x 40 entries out of 20 k columns, K = 16 / 32 / 52 / 128,
// 157 / 267 / 423 / 679 us against 672 / 674 / 676 / 691; 400 k x 16 out of 100 k 69 / 101 / 175 / 282 against
// 243 / 245 / 246 / 258.  Short rows with K > 64 and small matrices stay behind it (400 k x 5, K = 128, 150 us
// against 128; 20 k x 15, K = 128, 27.6 against 20.6): more row ends per entry, and a chain of searches before
// the first gather.
// A segment that holds a whole row stores it; the pieces of a cut row are added with vector
// reductions into `out`, cleared before by spmm_clear_kernel.
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

// STRAIGHT: batches of four entries inside one row skip the questions about row ends.
template <int G, bool TRANS, bool STRAIGHT>
__global__ void __launch_bounds__(256, STRAIGHT ? 5 : 0) spmm_kernel(const long long* __restrict__ row_ptr,
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
      if (STRAIGHT && p0 >= gs && p0 + U <= (end < ge ? end : ge)) {
#pragma unroll
        for (int j = 0; j < U; ++j)
          h[j] = on ? __ldg(reinterpret_cast<const float4*>(X + (long long)c[j] * K + 4 * gl)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < U; ++j) {
          acc.x = fmaf(v[j], h[j].x, acc.x); acc.y = fmaf(v[j], h[j].y, acc.y);
          acc.z = fmaf(v[j], h[j].z, acc.z); acc.w = fmaf(v[j], h[j].w, acc.w);
        }
        continue;
      }
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

// Zeros in the rows of `out` that spmm_kernel adds to (their entries lie in several segments of L) or
// does not touch (no entries).  Clearing all of `out` wrote it twice: 400 k rows x 5 entries, K = 128,
// 177 us, with this kernel 152.
__global__ void __launch_bounds__(256) spmm_clear_kernel(const long long* __restrict__ row_ptr, long long n_rows,
                                                         long long n_ent, int L, int K, float* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const long long r0 = ((long long)blockIdx.x * 256 + threadIdx.x) / 32 * 32, r = r0 + lane;
  bool zero = false;
  if (r < n_rows) {
    const long long b = __ldg(row_ptr + r), e = __ldg(row_ptr + r + 1);
    zero = e <= b || e > n_ent || ((b ^ (e - 1)) & ~(long long)(L - 1)) != 0;   // L is a power of two
  }
  for (unsigned todo = __ballot_sync(0xffffffffu, zero); todo; todo &= todo - 1) {
    float* o = out + (r0 + __ffs(todo) - 1) * K + 4 * lane;
    if (4 * lane < K) *reinterpret_cast<float4*>(o) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

template <bool TRANS>
int launch_spmm(const long long* row_ptr, const int* cols, const float* vals, long long n_rows,
                long long n_ent, const float* X, int K, float* out, cudaStream_t stream) {
  int G = 1;
  while (4 * G < K) G *= 2;
  // Entries per group: 128, fewer while the chip's groups (2048 threads on each of 148 SMs) would not all get a
  // segment.  From K = 36 on four times as many if that leaves four segments each (fewer row searches: 20 M
  // entries, K = 128, 724 us at 128 and 679 at 512), and fewer than 2 G only for a third of the groups (300 k
  // entries, K = 128: 27.6 us against 33.8).
  const bool wide = G >= 16 && !TRANS;
  int L = wide ? 512 : 128;
  while (L > 128 && n_ent / L < 4 * 148LL * 2048 / G) L /= 2;
  while (L > (wide ? 2 * G : 16) && n_ent / L < 148LL * 2048 / G) L /= 2;
  while (L > 16 && n_ent / L < 148LL * 640 / G) L /= 2;
  const long long blocks = (n_ent + (256 / G) * (long long)L - 1) / ((256 / G) * (long long)L);
  const long long clear = (n_rows + 255) / 256;
  if (blocks > 0x7fffffffLL || clear > 0x7fffffffLL) return (int)cudaErrorInvalidValue;
  if constexpr (!TRANS) {
    if (n_rows * K <= 1 << 22) {                   // up to 16 MB clearing all is up to 2 us faster
      const cudaError_t e = cudaMemsetAsync(out, 0, (size_t)n_rows * K * sizeof(float), stream);
      if (e != cudaSuccess) return (int)e;
    } else {
      spmm_clear_kernel<<<(int)clear, 256, 0, stream>>>(row_ptr, n_rows, n_ent, L, K, out);
    }
  }
  // Straight batches pay where a group is a warp (100 k rows x 200 entries, K = 128: 889 -> 693 us).  Where two groups
  // share one, a warp goes both ways unless rows are long: 100 k rows of up to 80 entries, K = 52, 113 -> 102 us,
  // of up to 30 entries 55 -> 59 us.  Narrower groups lose either way (400 k x 5, K = 32: 77 -> 83 us).
  const bool straight = G == 16 && n_ent >= 32 * n_rows;
#define PCL_SPMM(GG, ST)                                                                                       \
  spmm_kernel<GG, TRANS, ST><<<(int)blocks, 256, 0, stream>>>(row_ptr, cols, vals, n_rows, n_ent, L, X, K, out)
  switch (G) {
    case 1: PCL_SPMM(1, false); break;
    case 2: PCL_SPMM(2, false); break;
    case 4: PCL_SPMM(4, false); break;
    case 8: PCL_SPMM(8, false); break;
    case 16:
      if (straight) PCL_SPMM(16, !TRANS);
      else PCL_SPMM(16, false);
      break;
    case 32: PCL_SPMM(32, !TRANS); break;
  }
#undef PCL_SPMM
  return pcl_last_error();
}

// out = M P (TWICE: (M P) P^T) for M [n x K] and P [K x K], K a multiple of 4, fp32 throughout.  A
// block of 256 threads takes 128 rows at a time: thread (ty, tx) owns rows ty + 16 i (i < 8) and columns
// tx + 16 j, sums over even and odd components in the halves of packed multiply-adds.  P^T and, for
// the second product, P stay in shared memory as rows of components, and the product of the first
// takes the place of the rows there.  Bound by shared-memory passes: a thread loads 8 + KB times
// 16 bytes for 32 KB multiply-adds over four components.  The products of the SVD, 400 k x 32 and
// 100 k x 32 twice, take 83 and 29 us (86 and 31 with 4 rows a thread; at 400 k x 52 that form was faster, 199
// against 211 us, at 400 k x 112 slower, 715 against 643).
template <int KB, bool TWICE>
__global__ void __launch_bounds__(256) rows_times_kernel(const float* __restrict__ M, long long n, int K,
                                                         const float* __restrict__ P, float* __restrict__ out) {
  typedef unsigned long long u64;
  constexpr int N = 16 * KB, R = 128;    // columns padded with zeros; rows of a block
  extern __shared__ __align__(16) float sm[];
  const int LM = K + 4;                  // row pitch: eight rows of sixteen bytes on different banks
  float* sP = sm;                        // N x LM: column c of P
  float* sQ = sP + (TWICE ? N * LM : 0); // N x LM: row c of P
  float* sM = sQ + N * LM;               // R x LM
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  for (int e = tid; e < K * N; e += 256) {
    const int q = e / N, c = e % N;
    sP[c * LM + q] = c < K ? __ldg(P + q * K + c) : 0.f;
    if (TWICE) sQ[c * LM + q] = c < K ? __ldg(P + c * K + q) : 0.f;
  }
  const int K4 = K / 4;
  for (long long r0 = (long long)blockIdx.x * R; r0 < n; r0 += (long long)gridDim.x * R) {
    __syncthreads();
    for (int e = tid; e < R * K4; e += 256) {
      const int r = e / K4, c = 4 * (e % K4);
      *reinterpret_cast<float4*>(sM + r * LM + c) =
          r0 + r < n ? __ldg(reinterpret_cast<const float4*>(M + (r0 + r) * K + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
#pragma unroll
    for (int pass = 0; pass < (TWICE ? 2 : 1); ++pass) {
      const float* B = pass == 0 ? sP : sQ;
      u64 acc[8][KB];
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < KB; ++j) acc[i][j] = 0ull;
#pragma unroll 1
      for (int q = 0; q < K; q += 4) {
        ulonglong2 m[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) m[i] = *reinterpret_cast<const ulonglong2*>(sM + (ty + 16 * i) * LM + q);
#pragma unroll
        for (int j = 0; j < KB; ++j) {
          const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(B + (tx + 16 * j) * LM + q);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(m[i].x), "l"(b.x));
            asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(m[i].y), "l"(b.y));
          }
        }
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < KB; ++j) {
          float even, odd;
          asm("mov.b64 {%0, %1}, %2;" : "=f"(even), "=f"(odd) : "l"(acc[i][j]));
          if (tx + 16 * j < K) sM[(ty + 16 * i) * LM + tx + 16 * j] = even + odd;
        }
      __syncthreads();
    }
    for (int e = tid; e < R * K4; e += 256) {
      const int r = e / K4, c = 4 * (e % K4);
      if (r0 + r < n)
        *reinterpret_cast<float4*>(out + (r0 + r) * K + c) = *reinterpret_cast<const float4*>(sM + r * LM + c);
    }
  }
}

template <int KB, bool TWICE>
int launch_rows_times(const float* M, long long n, int K, const float* P, float* out, cudaStream_t stream) {
  const size_t smem = (16 * (size_t)KB * (TWICE ? 2 : 1) + 128) * (size_t)(K + 4) * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(rows_times_kernel<KB, TWICE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, rows_times_kernel<KB, TWICE>, 256, smem);
  if (e != cudaSuccess) return (int)e;
  long long blocks = (n + 127) / 128;
  const long long most = 148LL * (per_sm > 0 ? per_sm : 1);
  if (blocks > most) blocks = most;
  rows_times_kernel<KB, TWICE><<<(int)blocks, 256, smem, stream>>>(M, n, K, P, out);
  return pcl_last_error();
}

// out[i] = scale * u_i + shift with u_i = (word_i mod 2^24) / 2^24 for the words of the Mersenne Twister
// MT19937 (Matsumoto and Nishimura, 1998) after init_genrand(seed): the stream of the host
// generator, made where it is used.
// One block makes the words, in one chain of steps.  x[k + 624] = x[k + 397] ^ f(x[k], x[k + 1]) gives 227
// words a step; putting the recurrence in for x[k + 397] and again for x[k + 170] (f is linear),
//   x[k + 624] = x[k - 57] ^ f(x[k - 454] ^ x[k - 227] ^ x[k], x[k - 453] ^ x[k - 226] ^ x[k + 1]),
// gives 623, and a step costs little more than the barrier that ends it.  The words are tempered and
// scaled by a kernel of many blocks behind it.  3.2 M numbers took 1.5 ms with both in one block.
constexpr int MT_T = 640, MT_W = 623;

__device__ __forceinline__ unsigned mt_f(unsigned a, unsigned b) {
  const unsigned y = (a & 0x80000000u) | (b & 0x7fffffffu);
  return (y >> 1) ^ ((0u - (y & 1u)) & 0x9908b0dfu);
}

__global__ void __launch_bounds__(MT_T) mt19937_words_kernel(unsigned* __restrict__ out, long long n, unsigned seed) {
  __shared__ unsigned x[2048];           // word k at k mod 2048: a step reads 1078 back and writes 623
  const int t = threadIdx.x;
  if (t == 0) {
    unsigned s = seed;
    x[0] = s;
    for (int k = 1; k < 624; ++k) {
      s = 1812433253u * (s ^ (s >> 30)) + (unsigned)k;
      x[k] = s;
    }
  }
  __syncthreads();
  // words 624 .. 1077 by the recurrence itself: the long form reads 454 words before the state
  for (int k0 = 0; k0 < 454; k0 += 227) {
    if (t < 227) {
      const unsigned v = x[k0 + t + 397] ^ mt_f(x[k0 + t], x[k0 + t + 1]);
      x[k0 + t + 624] = v;
      if (k0 + t < n) out[k0 + t] = v;
    }
    __syncthreads();
  }
  for (long long i0 = 454; i0 < n; i0 += MT_W) {
    if (t < MT_W) {
      const int k = (int)((i0 + t) & 2047);
      auto w = [&](int d) { return x[(k + d) & 2047]; };
      const unsigned v = w(-57) ^ mt_f(w(-454) ^ w(-227) ^ w(0), w(-453) ^ w(-226) ^ w(1));
      x[(k + 624) & 2047] = v;
      if (i0 + t < n) out[i0 + t] = v;
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) mt19937_temper_kernel(float* out, long long n, float scale, float shift) {
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
    unsigned v = __float_as_uint(out[i]);
    v ^= v >> 11;
    v ^= (v << 7) & 0x9d2c5680u;
    v ^= (v << 15) & 0xefc60000u;
    v ^= v >> 18;
    out[i] = fmaf((float)(v & 0xffffffu) * (1.f / 16777216.f), scale, shift);
  }
}

// One CTA of CH_T threads.  Shared memory: L (K x K doubles) and X = L^-1 (K x K doubles).  Everything is a
// chain over the columns: two barriers a column in the factorisation, and a warp per column of the
// inverse that eliminates as it goes (with one thread per column and dot products, the first
// column's chain of K^2 / 2 dependent multiply-adds was most of 40 us at K = 32; 30 us now).
constexpr int CH_T = 512;

__global__ void __launch_bounds__(CH_T) chol_factor_kernel(const float* __restrict__ G, int K,
                                                           float* __restrict__ T, float* __restrict__ R,
                                                           double rel_tol, int* __restrict__ info) {
  extern __shared__ double sd[];
  double* L = sd;
  double* X = sd + (size_t)K * K;
  __shared__ double s_col[112], s_inv[112], s_max;
  const int tid = threadIdx.x, nt = CH_T, lane = tid & 31, warp = tid >> 5;
  for (int e = tid; e < K * K; e += nt) {
    const int i = e / K, j = e % K;
    L[e] = 0.5 * ((double)G[i * K + j] + (double)G[j * K + i]);   // symmetrise
  }
  __syncthreads();
  if (warp == 0) {
    double m = 0.0;
    for (int i = lane; i < K; i += 32) m = fmax(m, fabs(L[i * K + i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) s_max = m;
  }
  __syncthreads();
  // right-looking Cholesky on the lower triangle
  const double tol = rel_tol * s_max;
  const int tx = tid & 15, ty = tid >> 4;       // 16 columns x 32 rows of the trailing matrix
  for (int j = 0; j < K; ++j) {
    const double d = L[j * K + j];
    if (!(d > tol)) {                           // the same for every thread
      if (tid == 0) *info = j + 1;
      return;
    }
    // column j of the factor goes to a buffer of its own: its place is read by the threads still here
    const double inv = 1.0 / sqrt(d);
    if (tid == 0) s_inv[j] = inv;
    for (int i = j + tid; i < K; i += nt) s_col[i] = i == j ? d * inv : L[i * K + j] * inv;
    __syncthreads();
    for (int i = j + tid; i < K; i += nt) L[i * K + j] = s_col[i];
    for (int i = j + 1 + ty; i < K; i += CH_T / 16)
      for (int k = j + 1 + tx; k <= i; k += 16) L[i * K + k] -= s_col[i] * s_col[k];
    __syncthreads();
  }
  // X = L^-1, a warp per column: lane l holds rows l, l + 32, ... of the column
  for (int c = warp; c < K; c += nt / 32) {
    double b[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) b[q] = lane + 32 * q == c ? 1.0 : 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      for (int l = 0; l < 32; ++l) {
        const int k = 32 * q + l;
        if (k >= K) break;
        if (k < c) continue;
        const double x = __shfl_sync(0xffffffffu, b[q], l) * s_inv[k];
        if (lane == l) b[q] = x;
#pragma unroll
        for (int p = q; p < 4; ++p) {
          const int i = lane + 32 * p;
          if (i > k && i < K) b[p] -= L[i * K + k] * x;
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (lane + 32 * q < K) X[(lane + 32 * q) * K + c] = lane + 32 * q >= c ? b[q] : 0.0;
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
  if (n_ent <= 0) return (int)cudaMemsetAsync(out, 0, (size_t)n_rows * K * sizeof(float), stream);
  return launch_spmm<false>(row_ptr, cols, vals, n_rows, n_ent, H, K, out, stream);
}

PCL_API int pcl_spmm_csr_t(const long long* row_ptr, const int* cols, const float* vals, long long n_rows,
                           long long n_ent, const float* W, int K, float* out, cudaStream_t stream) {
  if (n_rows <= 0 || n_ent <= 0) return 0;
  if (K <= 0 || K > 128 || (K & 3)) return (int)cudaErrorInvalidValue;
  return launch_spmm<true>(row_ptr, cols, vals, n_rows, n_ent, W, K, out, stream);
}

// M and out 16-byte aligned, K <= 112 a multiple of 4; twice: out = (M P) P^T, else M P.
PCL_API int pcl_rows_times(const float* M, long long n, int K, const float* P, int twice, float* out,
                           cudaStream_t stream) {
  if (n <= 0) return 0;
  if (K <= 0 || K > 112 || (K & 3)) return (int)cudaErrorInvalidValue;
#define PCL_RT(KB)                                                                    \
  case KB:                                                                            \
    return twice ? launch_rows_times<KB, true>(M, n, K, P, out, stream)               \
                 : launch_rows_times<KB, false>(M, n, K, P, out, stream);
  switch ((K + 15) / 16) {
    PCL_RT(1) PCL_RT(2) PCL_RT(3) PCL_RT(4) PCL_RT(5) PCL_RT(6) PCL_RT(7)
  }
#undef PCL_RT
  return (int)cudaErrorInvalidValue;
}

PCL_API int pcl_mt19937_uniform(float* out, long long n, unsigned int seed, float scale, float shift,
                                cudaStream_t stream) {
  if (n <= 0) return 0;
  mt19937_words_kernel<<<1, MT_T, 0, stream>>>(reinterpret_cast<unsigned*>(out), n, seed);
  const long long need = (n + 255) / 256;
  mt19937_temper_kernel<<<need < 148 * 8 ? (int)need : 148 * 8, 256, 0, stream>>>(out, n, scale, shift);
  return pcl_last_error();
}

PCL_API int pcl_chol_factor(const float* G, int K, float* T, float* R, double rel_tol, int* info,
                            cudaStream_t stream) {
  if (K <= 0 || K > 112) return (int)cudaErrorInvalidValue;   // 2 K^2 doubles must fit in 227 KB
  const size_t smem = 2 * (size_t)K * K * sizeof(double);
  cudaError_t e = cudaFuncSetAttribute(chol_factor_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return (int)e;
  chol_factor_kernel<<<1, CH_T, smem, stream>>>(G, K, T, R, rel_tol, info);
  return pcl_last_error();
}
