// Smaller kernels of the algorithm suite.
//   kmeans_accumulate  per-cluster sums and counts after the assignment GEMM
//                      (alg/clustering/kmeans/kmeans.hpp:127-133)
//   topk_rows          running per-row top-k of a similarity tile with a lower bound and
//                      self-exclusion (alg/recommendation/similarity_dense/sim_dense.hpp:84-101)
//   gram               H^T H of a tall-skinny block (alg/recommendation/svd/svd.hpp:137-148)
//   allreduce_sum      sum of a small vector over all ranks through peer memory (the
//                      MPI_Allreduce of loss / RMSE / likelihood scalars, lr.cpp:331-334,
//                      mf.hpp:104-106), one launch, bounded wait
#include <cuda_pipeline.h>

#include "common.cuh"

namespace {

__global__ void __launch_bounds__(256) kmeans_accumulate_kernel(const float* X, const int* assign,
                                                                long long n, int d, float* sums,
                                                                float* counts) {
  const int lane = threadIdx.x & 31;
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long i = warp; i < n; i += nwarps) {
    const int c = assign[i];
    const float* x = X + i * d;
    float* s = sums + (long long)c * d;
    for (int j = lane; j < d; j += 32) atomicAdd(s + j, x[j]);
    if (lane == 0) atomicAdd(counts + c, 1.f);
  }
}

// d a multiple of 4 and at most 512, X and sums 16-byte aligned: a lane owns up to four 16-byte
// pieces of a row and adds each with one vector reduction (a quarter of the requests the L2 atomic
// units see with scalar adds).  A warp takes four points per step: the four cluster ids, then all
// row pieces, then the reductions, so four rows are in flight per warp instead of one.
template <int PIECES>
__global__ void __launch_bounds__(256) kmeans_accumulate_vec_kernel(const float* X, const int* assign,
                                                                    long long n, int d, float* sums,
                                                                    float* counts) {
  constexpr int P = 4;
  const int lane = threadIdx.x & 31;
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long i0 = warp * P; i0 < n; i0 += nwarps * P) {
    int c[P];
#pragma unroll
    for (int k = 0; k < P; ++k) c[k] = (i0 + k < n) ? __ldg(assign + i0 + k) : -1;
    float4 x[P][PIECES];
#pragma unroll
    for (int k = 0; k < P; ++k)
#pragma unroll
      for (int q = 0; q < PIECES; ++q) {
        const int j = (q * 32 + lane) * 4;
        if (c[k] >= 0 && j < d) x[k][q] = __ldcs(reinterpret_cast<const float4*>(X + (i0 + k) * d + j));
      }
#pragma unroll
    for (int k = 0; k < P; ++k) {
      if (c[k] < 0) continue;
      float* s = sums + (long long)c[k] * d;
#pragma unroll
      for (int q = 0; q < PIECES; ++q) {
        const int j = (q * 32 + lane) * 4;
        if (j < d)
          asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(s + j), "f"(x[k][q].x),
                       "f"(x[k][q].y), "f"(x[k][q].z), "f"(x[k][q].w)
                       : "memory");
      }
      if (lane == 0) atomicAdd(counts + c[k], 1.f);
    }
  }
}

// Few clusters: the reductions above all go to a few addresses (900 k points of 8 columns in 10 clusters
// took 1.19 ms, now 13 us; of 100 columns in 12 clusters 1.41 ms, now 70 us).  Here every group of LG lanes that takes a
// point at a time has sums of its own in shared memory, plain additions without atomics, and a block
// adds its copies up at the end.  A lane owns PIECES 16-byte pieces of a row; four points are in
// flight per group.
template <int LG, int PIECES>
__global__ void kmeans_accumulate_few_kernel(const float* X, const int* assign, long long n, int d, int k,
                                             int copy_floats, float* sums, float* counts) {
  constexpr int U = 4;
  extern __shared__ __align__(16) float s_c[];     // copies x (k x d sums, k counts)
  const int groups = blockDim.x / LG, grp = threadIdx.x / LG, l = threadIdx.x % LG;
  for (int e = threadIdx.x; e < groups * copy_floats; e += blockDim.x) s_c[e] = 0.f;
  __syncthreads();
  float* mine = s_c + grp * copy_floats;
  const long long step = (long long)gridDim.x * groups;
  for (long long i0 = (long long)blockIdx.x * groups + grp; i0 < n; i0 += U * step) {
    int c[U];
    float4 x[U][PIECES];
#pragma unroll
    for (int u = 0; u < U; ++u) c[u] = i0 + u * step < n ? __ldg(assign + i0 + u * step) : -1;
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int q = 0; q < PIECES; ++q) {
        const int j = 4 * (q * LG + l);
        if (i0 + u * step < n && j < d) x[u][q] = __ldcs(reinterpret_cast<const float4*>(X + (i0 + u * step) * d + j));
      }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (c[u] < 0 || c[u] >= k) continue;
#pragma unroll
      for (int q = 0; q < PIECES; ++q) {
        const int j = 4 * (q * LG + l);
        if (j < d) {
          float4* p = reinterpret_cast<float4*>(mine + c[u] * d + j);
          float4 v = *p;
          v.x += x[u][q].x; v.y += x[u][q].y; v.z += x[u][q].z; v.w += x[u][q].w;
          *p = v;
        }
      }
      if (l == 0) mine[k * d + c[u]] += 1.f;
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < k * d + k; e += blockDim.x) {
    float v = 0.f;
    for (int g = 0; g < groups; ++g) v += s_c[g * copy_floats + e];
    if (v != 0.f) atomicAdd(e < k * d ? sums + e : counts + (e - k * d), v);
  }
}

// Warps of a block of kmeans_accumulate_few_kernel; 0: the clusters are too many.  Six groups per SM beat
// the reductions (500 k points: 64 columns in 100 clusters 235 -> 171 us, 128 in 64 362 -> 174 us),
// three did not (128 in 120: 324 against 336 us).
inline int km_few_warps(long long copy_bytes, int groups_per_warp) {
  if (copy_bytes <= 100 * 1024 / 3) return (int)(100 * 1024 / copy_bytes < 8 ? 100 * 1024 / copy_bytes : 8);
  const int w = (int)(200 * 1024 / copy_bytes);
  return w * groups_per_warp >= 5 ? w : 0;
}

// Clearing and adding up a block's own sums takes a time that grows with k, and more with wide rows,
// whose sums leave room for fewer warps; the reductions queue up for n / k of them per address.  The line
// fits both sides measured at 10 k, 100 k and 900 k points of 4 to 512 columns in 2 to 200 clusters: 10 k x 8 in 30
// clusters 14.4 us with reductions against 10.3 here, in 64 12.3 against 14.3, in 200 11 against 32;
// 100 k x 64 in 64 83 against 37, in 100 52 against 56; 100 k x 16 in 120 43 against 29, in 200 32 against 47.
inline bool km_few_pays(long long n, int d, int k) {
  const long long w = d > 128 || d < 68 ? 20 + d : 88;
  return k < 1 << 16 && (long long)k * k * w <= 8 * n;
}

template <int LG, int PIECES>
int launch_km_few(const float* X, const int* assign, long long n, int d, int k, float* sums, float* counts,
                  bool* taken, cudaStream_t stream) {
  const long long copy_floats = ((long long)k * (d + 1) + 3) / 4 * 4;
  const int warps = km_few_warps(copy_floats * 4 * (32 / LG), 32 / LG);
  *taken = warps > 0;
  if (warps == 0) return 0;
  auto kernel = kmeans_accumulate_few_kernel<LG, PIECES>;
  const size_t smem = (size_t)copy_floats * 4 * (32 / LG) * warps;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 32 * warps, smem);
  if (e != cudaSuccess) return (int)e;
  const long long per_block = (long long)warps * (32 / LG) * 4;
  long long blocks = (n + per_block - 1) / per_block;
  if (blocks > 148LL * (per_sm > 0 ? per_sm : 1)) blocks = 148LL * (per_sm > 0 ? per_sm : 1);
  kernel<<<(int)blocks, 32 * warps, smem, stream>>>(X, assign, n, d, k, (int)copy_floats, sums, counts);
  return pcl_last_error();
}

// Lane i of the warp holds the i-th best (value, id) of its row, best first.  Bound by reading S
// once: a warp asks for TK_U x 128 columns before it looks at the first (2 KB in flight per warp, with
// 32 columns at a time the scan of a row was a chain of load latencies), and the 8-byte column ids,
// twice the size of the row itself, are read for candidates only.
// Measured on 12,007 x 12,007, k = 20: 0.46 -> 0.24 ms; most of what is left are the ~150 insertions
// of a row, each a chain of ballots and shuffles.
constexpr int TK_U = 4;
constexpr float TK_NONE = -3.402823466e38f;

// VEC: rows start on 16-byte boundaries and a lane takes columns 4 lane .. 4 lane + 3 of a group of
// 128; otherwise it takes columns 32 t + lane.  Candidates are taken in column order in both
// layouts, so that of two equal values the lower column stays ahead.
template <bool VEC>
__global__ void __launch_bounds__(256) topk_rows_kernel(const float* S, long long ldS, int m, int n,
                                                        const long long* row_ids,
                                                        const long long* col_ids, float lower, int k,
                                                        float* best_val, long long* best_idx) {
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int r = warp; r < m; r += nwarps) {
    float v = TK_NONE;
    long long id = -1;
    if (lane < k) { v = best_val[(long long)r * k + lane]; id = best_idx[(long long)r * k + lane]; }
    const long long self = row_ids ? row_ids[r] : -1;
    const float* row = S + (long long)r * ldS;
    float kth = __shfl_sync(0xffffffffu, v, k - 1);
    auto insert = [&](float xv, long long xi) {      // warp-uniform arguments
      if (!(xv > kth)) return;
      // position = number of entries that stay ahead of the newcomer
      const int pos = __popc(__ballot_sync(0xffffffffu, lane < k && v >= xv));
      const float vup = __shfl_up_sync(0xffffffffu, v, 1);
      const long long iup = __shfl_up_sync(0xffffffffu, id, 1);
      if (lane > pos && lane < k) { v = vup; id = iup; }
      if (lane == pos) { v = xv; id = xi; }
      kth = __shfl_sync(0xffffffffu, v, k - 1);
    };
    for (int c0 = 0; c0 < n; c0 += 128 * TK_U) {
      float x[TK_U][4];
#pragma unroll
      for (int q = 0; q < TK_U; ++q) {
        const int b = c0 + 128 * q;
        if (VEC && b + 4 * lane + 3 < n) {
          const float4 f = __ldcs(reinterpret_cast<const float4*>(row + b + 4 * lane));
          x[q][0] = f.x; x[q][1] = f.y; x[q][2] = f.z; x[q][3] = f.w;
        } else {
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const int c = b + (VEC ? 4 * lane + t : 32 * t + lane);
            x[q][t] = c < n ? __ldcs(row + c) : TK_NONE;
          }
        }
      }
#pragma unroll
      for (int q = 0; q < TK_U; ++q) {
        const int b = c0 + 128 * q;
        unsigned mine = 0;                           // bit t: x[q][t] may enter the heap
#pragma unroll
        for (int t = 0; t < 4; ++t)
          if (x[q][t] >= lower && x[q][t] > kth) mine |= 1u << t;
        if (__ballot_sync(0xffffffffu, mine != 0) == 0) continue;
        long long cid[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int c = b + (VEC ? 4 * lane + t : 32 * t + lane);
          cid[t] = -1;
          if ((mine >> t) & 1) {
            if (c < n) cid[t] = col_ids ? __ldg(col_ids + c) : c;
            if (c >= n || cid[t] == self) mine &= ~(1u << t);
          }
        }
        if (VEC) {
          unsigned cand = __ballot_sync(0xffffffffu, mine != 0);
          while (cand) {
            const int src = __ffs(cand) - 1;
            cand &= cand - 1;
            const unsigned bits = __shfl_sync(0xffffffffu, mine, src);
#pragma unroll
            for (int t = 0; t < 4; ++t)
              if ((bits >> t) & 1)
                insert(__shfl_sync(0xffffffffu, x[q][t], src), __shfl_sync(0xffffffffu, cid[t], src));
          }
        } else {
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            unsigned cand = __ballot_sync(0xffffffffu, (mine >> t) & 1);
            while (cand) {
              const int src = __ffs(cand) - 1;
              cand &= cand - 1;
              insert(__shfl_sync(0xffffffffu, x[q][t], src), __shfl_sync(0xffffffffu, cid[t], src));
            }
          }
        }
      }
    }
    if (lane < k) { best_val[(long long)r * k + lane] = v; best_idx[(long long)r * k + lane] = id; }
  }
}

// H^T H over the lower triangle: a warp owns a 32 x 32 block of it, 4 x 8 values per lane as pairs for the
// packed multiply-add; with fewer than ten blocks several warps share one and split the rows.  A row
// costs a warp three 16-byte shared-memory loads (12 passes) for 1024 multiply-adds; with 2 x 2
// values per thread of one 16 x 16 grid it took 32 passes (mean of 400 k x 32 and 100 k x 32: 52 -> 36 us).
// Rows arrive by asynchronous copies one stage ahead.  For k > 64, where one group takes all rows of
// a block, the registers' sums go to shared memory after GM_RUN rows: rounding errors grow with the length
// of a chain of additions (3 M x 128: relative error 4.7e-7 without that, 2.5e-7 with it).
constexpr int GM_T = 320, GM_RS = 40, GM_RUN = 1280;

template <int KB>
__global__ void __launch_bounds__(GM_T) gram_kernel(const float* H, long long n, int k, int vec, float* out) {
  constexpr int K = 16 * KB, B = KB / 2, NB = B * (B + 1) / 2, GR = 10 / NB;
  extern __shared__ __align__(16) float sm[];      // two stages of GM_RS x K rows, then the groups' K x K sums
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int blk = warp % NB, grp = warp / NB;
  const bool has_blk = grp < GR;
  int bi = 0;
  while ((bi + 1) * (bi + 2) / 2 <= blk) ++bi;
  const int bj = blk - bi * (bi + 1) / 2;
  const int row0 = 32 * bi + 4 * (lane >> 2), col0 = 32 * bj + 4 * (lane & 3);
  typedef unsigned long long u64;
  auto pack = [](float x) {
    u64 r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
    return r;
  };
  auto fma2 = [](u64 x, u64 y, u64 z) {
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(z));
    return r;
  };
  u64 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
  for (int e = tid; e < 2 * GM_RS * K; e += GM_T) sm[e] = 0.f;   // columns behind k stay zero
  __syncthreads();
  const long long stages = (n + GM_RS - 1) / GM_RS;
  auto stage = [&](long long s, int buf) {
    if (s < stages) {
      float* dst = sm + buf * GM_RS * K;
      const long long r0 = s * GM_RS;
      for (int r = warp; r < GM_RS; r += GM_T / 32) {
        const bool in = r0 + r < n;                // rows past the end: zeros
        const float* src = H + (in ? r0 + r : 0) * k;
        if (vec) {
          if (4 * lane < k) __pipeline_memcpy_async(dst + r * K + 4 * lane, src + 4 * lane, 16, in ? 0 : 16);
        } else {
          for (int c = lane; c < k; c += 32) __pipeline_memcpy_async(dst + r * K + c, src + c, 4, in ? 0 : 4);
        }
      }
    }
    __pipeline_commit();
  };
  float* sS = sm + 2 * GM_RS * K + (has_blk ? grp : 0) * K * K;   // sums of this warp's group
  bool fresh = true;
  auto add_up = [&]() {                            // the registers' sums into shared memory
    if (has_blk) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float v[2];
          asm("mov.b64 {%0, %1}, %2;" : "=f"(v[0]), "=f"(v[1]) : "l"(acc[i][j]));
          acc[i][j] = 0ull;
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            float* p = sS + (row0 + i) * K + col0 + 16 * (j >> 1) + 2 * (j & 1) + q;
            *p = fresh ? v[q] : *p + v[q];
          }
        }
    }
    fresh = false;
  };
  int buf = 0, since = 0;
  stage(blockIdx.x, 0);
  for (long long s = blockIdx.x; s < stages; s += gridDim.x, buf ^= 1) {
    stage(s + gridDim.x, buf ^ 1);
    __pipeline_wait_prior(1);
    __syncthreads();
    const float* sh = sm + buf * GM_RS * K;
    if (has_blk) {
#pragma unroll 4
      for (int r = grp; r < GM_RS; r += GR) {
        const float4 h = *reinterpret_cast<const float4*>(sh + r * K + row0);
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(sh + r * K + col0);
        const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(sh + r * K + col0 + 16);
        const u64 hh[4] = {pack(h.x), pack(h.y), pack(h.z), pack(h.w)};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc[i][0] = fma2(hh[i], x.x, acc[i][0]);
          acc[i][1] = fma2(hh[i], x.y, acc[i][1]);
          acc[i][2] = fma2(hh[i], y.x, acc[i][2]);
          acc[i][3] = fma2(hh[i], y.y, acc[i][3]);
        }
      }
    }
    __syncthreads();
    if (GR == 1 && ++since == GM_RUN / GM_RS) {
      since = 0;
      add_up();
    }
  }
  __pipeline_wait_prior(0);
  add_up();
  __syncthreads();
  const float* all = sm + 2 * GM_RS * K;
  for (int e = tid; e < k * k; e += GM_T) {
    const int r = e / k, c = e % k;
    const float* p = all + (c <= r ? r * K + c : c * K + r);
    float v = p[0];
#pragma unroll
    for (int g = 1; g < GR; ++g) v += p[g * K * K];
    if (v != 0.f) atomicAdd(out + e, v);
  }
}

template <int KB>
int launch_gram(const float* H, long long n, int k, float* out, cudaStream_t stream) {
  constexpr int B = KB / 2, GR = 10 / (B * (B + 1) / 2);          // as in the kernel
  const size_t smem = (2 * (size_t)GM_RS * 16 * KB + GR * 256 * (size_t)KB * KB) * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(gram_kernel<KB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const long long need = (n + 63) / 64;            // every block's sums are one more addition per entry
  const int blocks = need < 148 * 2 ? (int)need : 148 * 2;
  const int vec = (k & 3) == 0 && (reinterpret_cast<uintptr_t>(H) & 15) == 0;
  gram_kernel<KB><<<blocks, GM_T, smem, stream>>>(H, n, k, vec, out);
  return pcl_last_error();
}

struct ArArgs {
  const double* in;          // n values of this rank
  double* out;               // n sums
  int n;
  double* const* slots;      // world pointers: each rank's 2 x nmax staging area
  long long* const* flags;   // world pointers: each rank's flag array (world entries)
  const long long* my_flags; // this rank's flag array
  int world, rank, nmax;
  long long epoch;
  unsigned long long timeout_ns;
  PclStatus* status;
};

__global__ void __launch_bounds__(256) allreduce_sum_kernel(ArArgs a) {
  __shared__ int ok;
  const int par = (int)(a.epoch & 1);
  double* mine = a.slots[a.rank] + (long long)par * a.nmax;
  for (int i = threadIdx.x; i < a.n; i += blockDim.x) mine[i] = a.in[i];
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x < a.world) pcl_st_release_sys(a.flags[threadIdx.x] + a.rank, a.epoch);
  if (threadIdx.x == 0)
    ok = pcl_wait_min_clock(a.my_flags, a.world, a.epoch, a.timeout_ns, a.status, a.rank, 30) ? 1 : 0;
  __syncthreads();
  if (!ok) return;
  for (int i = threadIdx.x; i < a.n; i += blockDim.x) {
    double s = 0.0;
    for (int r = 0; r < a.world; ++r) {
      double v;
      asm volatile("ld.relaxed.sys.global.f64 %0, [%1];" : "=d"(v) : "l"(a.slots[r] + (long long)par * a.nmax + i));
      s += v;
    }
    a.out[i] = s;
  }
}

}  // namespace

PCL_API int pcl_kmeans_accumulate(const float* X, const int* assign, long long n, int d, int k, float* sums,
                                  float* counts, cudaStream_t stream) {
  if (n <= 0) return 0;
  long long blocks = (n + 7) / 8;
  if (blocks > 148 * 8) blocks = 148 * 8;
  const bool vec = (d % 4 == 0) && d <= 512 && (((uintptr_t)X | (uintptr_t)sums) & 15) == 0;
  if (vec && k > 0 && km_few_pays(n, d, k)) {
    bool taken = false;
    int rc;
    if (d <= 4) rc = launch_km_few<1, 1>(X, assign, n, d, k, sums, counts, &taken, stream);
    else if (d <= 8) rc = launch_km_few<2, 1>(X, assign, n, d, k, sums, counts, &taken, stream);
    else if (d <= 16) rc = launch_km_few<4, 1>(X, assign, n, d, k, sums, counts, &taken, stream);
    else if (d <= 32) rc = launch_km_few<8, 1>(X, assign, n, d, k, sums, counts, &taken, stream);
    else if (d <= 64) rc = launch_km_few<16, 1>(X, assign, n, d, k, sums, counts, &taken, stream);
    else if (d <= 128) rc = launch_km_few<32, 1>(X, assign, n, d, k, sums, counts, &taken, stream);
    else if (d <= 256) rc = launch_km_few<32, 2>(X, assign, n, d, k, sums, counts, &taken, stream);
    else rc = launch_km_few<32, 4>(X, assign, n, d, k, sums, counts, &taken, stream);
    if (rc != 0 || taken) return rc;
  }
  if (vec) {
    blocks = (n + 31) / 32;
    if (blocks > 148 * 8) blocks = 148 * 8;
    if (d <= 128) kmeans_accumulate_vec_kernel<1><<<(int)blocks, 256, 0, stream>>>(X, assign, n, d, sums, counts);
    else if (d <= 256) kmeans_accumulate_vec_kernel<2><<<(int)blocks, 256, 0, stream>>>(X, assign, n, d, sums, counts);
    else kmeans_accumulate_vec_kernel<4><<<(int)blocks, 256, 0, stream>>>(X, assign, n, d, sums, counts);
  } else {
    kmeans_accumulate_kernel<<<(int)blocks, 256, 0, stream>>>(X, assign, n, d, sums, counts);
  }
  return pcl_last_error();
}

// best_val (m x k, initialised to -FLT_MAX) / best_idx (m x k, -1) are updated with the columns
// of the tile S (m x n, leading dimension ldS); k <= 32.
PCL_API int pcl_topk_rows(const float* S, long long ldS, int m, int n, const long long* row_ids,
                          const long long* col_ids, float lower, int k, float* best_val,
                          long long* best_idx, cudaStream_t stream) {
  if (m <= 0 || n <= 0) return 0;
  if (k <= 0 || k > 32) return (int)cudaErrorInvalidValue;
  int blocks = (m + 7) / 8;
  if (blocks > 148 * 8) blocks = 148 * 8;
  // 16-byte loads where every row starts on a 16-byte boundary
  if ((ldS & 3) == 0 && (reinterpret_cast<uintptr_t>(S) & 15) == 0)
    topk_rows_kernel<true><<<blocks, 256, 0, stream>>>(S, ldS, m, n, row_ids, col_ids, lower, k, best_val, best_idx);
  else
    topk_rows_kernel<false><<<blocks, 256, 0, stream>>>(S, ldS, m, n, row_ids, col_ids, lower, k, best_val, best_idx);
  return pcl_last_error();
}

// out (k x k, accumulated into; zero it first) += H^T H for H [n x k], k <= 128.
PCL_API int pcl_gram(const float* H, long long n, int k, float* out, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (k <= 0 || k > 128) return (int)cudaErrorInvalidValue;
  if (k <= 32) return launch_gram<2>(H, n, k, out, stream);
  if (k <= 64) return launch_gram<4>(H, n, k, out, stream);
  if (k <= 96) return launch_gram<6>(H, n, k, out, stream);
  return launch_gram<8>(H, n, k, out, stream);
}

PCL_API int pcl_allreduce_sum_f64(const double* in, double* out, int n, double* const* slots,
                                  long long* const* flags, const long long* my_flags, int world,
                                  int rank, int nmax, long long epoch, unsigned long long timeout_ns,
                                  PclStatus* status, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (n > nmax || world > 256) return (int)cudaErrorInvalidValue;
  ArArgs a{in, out, n, slots, flags, my_flags, world, rank, nmax, epoch, timeout_ns, status};
  allreduce_sum_kernel<<<1, 256, 0, stream>>>(a);
  return pcl_last_error();
}

// ---------------------------------------------------------------------------------------------
// Range check of an id array that a later kernel will use as an index without looking at it
// again (rating streams, CSR column arrays, word ids, topic assignments): run once when the
// data is loaded.  The first id outside [lo, hi) is recorded in the status block (code 2,
// wait_id 110, expected = position, seen = id); `skip` is a value that is allowed although it
// is out of range (padding markers), pass lo to allow none.
namespace {
template <typename T>
__global__ void validate_ids_kernel(const T* ids, long long n, long long lo, long long hi,
                                    long long skip, PclStatus* st, int rank) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const long long g = (long long)ids[i];
    if ((g < lo || g >= hi) && g != skip) pcl_report_bad_id(st, rank, 110, i, g);
  }
}
}  // namespace

PCL_API int pcl_validate_ids(const void* ids, int is64, long long n, long long lo, long long hi,
                             long long skip, PclStatus* status, int rank, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (status == nullptr) return (int)cudaErrorInvalidValue;
  long long blocks = (n + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  if (is64)
    validate_ids_kernel<long long><<<(int)blocks, 256, 0, stream>>>(
        static_cast<const long long*>(ids), n, lo, hi, skip, status, rank);
  else
    validate_ids_kernel<int><<<(int)blocks, 256, 0, stream>>>(static_cast<const int*>(ids), n, lo,
                                                              hi, skip, status, rank);
  return pcl_last_error();
}
