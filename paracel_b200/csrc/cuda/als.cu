// Batched ALS normal equations: for every user u with rated items I_u and ratings a_u,
//   w_u = (H_u^T H_u + lambda I)^-1 H_u^T a_u
// (reference: alg/recommendation/als/als.hpp:133-165, which forms the k x k matrix with Eigen
// and multiplies by its explicit inverse).
//
// Ratings per user are heavy-tailed, so a user takes one of three forms, chosen by its number of
// ratings n against the rank k (als_plan_kernel):
//   n <= 32, n < k     a warp solves the n x n system of the dual form
//                        w = H_u^T (H_u H_u^T + lambda I)^-1 a_u,
//                      the same vector for lambda > 0 from a far smaller matrix
//   n <= 96, n < k     a CTA solves the dual form in shared memory
//   otherwise          a CTA per segment of ratings forms the k x k matrix; a user with more than
//                      `split` ratings has several segments, which add their parts in a scratch
//                      slot, and the last one to arrive solves
// The dual form needs lambda > 0 (with lambda <= 0 every user takes the last form).
// Rank 128, 100 k users, 10 M Zipf(1.1) ratings: 84 % of the users have at most 32 ratings and
// 4.6 % more than 128, while those hold 82 % of the ratings; a solve takes 6.5 ms against 36.1 ms
// with the k x k form for everyone, of which two thirds were its 128 x 128 factorisations.
#include <cuda_pipeline.h>

#include "common.cuh"

namespace {

constexpr int NT = 192;            // threads of a CTA: six warps (six 32 x 64 blocks cover a 128 x 128 triangle)
constexpr int RS = 24;             // item rows per stage of the Gram loop, four per warp

// lists and counters the plan kernel writes
enum { C_BIG = 0, C_SMALL = 1, C_SLOT = 2, C_T16 = 3, C_T32 = 4, C_T64 = 5, C_T96 = 6, C_TICKET = 7, C_N = 8 };

struct AlsArgs {
  const long long* user_ptr;       // n_users + 1
  const int* item_idx;             // nnz: row of H
  const float* rating;             // nnz
  const float* H;                  // n_items x k
  float* W;                        // n_users x k (output; users without ratings are left alone)
  float* scratch;                  // slots x (K*K + K)
  int* slot_count;                 // slots: segments that have arrived
  int* counters;                   // C_N, zero on entry of the plan kernel
  int* seg_user;                   // seg_cap: long segments from the front, short ones from the back
  int* seg_piece;                  // seg_cap: which piece of the user's ratings
  int* seg_slot;                   // seg_cap: scratch slot of a split user, -1 otherwise
  int* user_list;                  // 4 x n_users: users of the dual forms (n <= 16, 32, 64, 96)
  long long n_users;
  long long split;                 // users with more ratings are cut into pieces of `piece`
  int piece;
  int seg_cap;
  int k;
  float lambda;
  int vec;                         // rows of H start on 16-byte boundaries and k is a multiple of 4
};

// Two fp32 multiply-adds in one instruction.  The fp32 pipe takes as long for one as for two: the Gram
// loop below took 5.9 ms with scalar multiply-adds and 4.9 ms with these (rank 128, 8.5 M ratings).
typedef unsigned long long u64;
__device__ __forceinline__ u64 pack2(float x, float y) {
  u64 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void unpack2(u64 v, float& x, float& y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
  u64 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// ------------------------------------------------------------------------------------------ plan
__global__ void __launch_bounds__(256) als_plan_kernel(AlsArgs a) {
  const long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= a.n_users) return;
  const long long n = a.user_ptr[u + 1] - a.user_ptr[u];
  if (n <= 0) return;
  if (a.lambda > 0.f && n < a.k && n <= 96) {
    const int cls = n <= 16 ? 0 : (n <= 32 ? 1 : (n <= 64 ? 2 : 3));
    a.user_list[cls * a.n_users + atomicAdd(a.counters + C_T16 + cls, 1)] = (int)u;
    return;
  }
  if (n <= a.split) {
    const bool big = n >= 512;     // long segments are handed out first: a short tail at the end
    const int p = atomicAdd(a.counters + (big ? C_BIG : C_SMALL), 1);
    const int at = big ? p : a.seg_cap - 1 - p;
    a.seg_user[at] = (int)u;
    a.seg_piece[at] = 0;
    a.seg_slot[at] = -1;
    return;
  }
  const int ns = (int)((n + a.piece - 1) / a.piece);
  const int slot = atomicAdd(a.counters + C_SLOT, 1);
  const int p = atomicAdd(a.counters + C_BIG, ns);
  a.slot_count[slot] = 0;
  for (int s = 0; s < ns; ++s) {
    a.seg_user[p + s] = (int)u;
    a.seg_piece[p + s] = s;
    a.seg_slot[p + s] = slot;
  }
}

__global__ void __launch_bounds__(256) als_clear_kernel(float* scratch, const int* counters, long long per_slot) {
  const long long n = counters[C_SLOT] * per_slot / 4;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    reinterpret_cast<float4*>(scratch)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// Row `src` of H (k floats) into shared memory by one warp; src null: zeros.
__device__ __forceinline__ void stage_row(float* dst, const float* src, const float* H, int k, int vec, int lane) {
  if (vec) {
    if (4 * lane < k) __pipeline_memcpy_async(dst + 4 * lane, (src ? src : H) + 4 * lane, 16, src ? 0 : 16);
  } else {
    for (int c = lane; c < k; c += 32) __pipeline_memcpy_async(dst + c, (src ? src : H) + c, 4, src ? 0 : 4);
  }
}

// ------------------------------------------------------------------- factorisation of one system
// 16 x 16 diagonal block at (j0, j0): its Cholesky factor in place, the inverse diagonal in s_inv.
// One warp; lane i (and i + 16) holds row i in registers, a column travels by shuffles.
__device__ __forceinline__ void diag_factor(float* sA, int LD, float* s_inv, int j0, int lane) {
  const int i = lane & 15;
  float a[16];
#pragma unroll
  for (int c = 0; c < 16; ++c) a[c] = c <= i ? sA[(j0 + i) * LD + j0 + c] : 0.f;
  float myinv = 0.f;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const float d = sqrtf(fmaxf(__shfl_sync(0xffffffffu, a[j], j), 1e-30f));
    const float inv = 1.f / d;
    const float l = i == j ? d : a[j] * inv;
    a[j] = l;
    if (i == j) myinv = inv;
#pragma unroll
    for (int c = j + 1; c < 16; ++c) a[c] = fmaf(-l, __shfl_sync(0xffffffffu, l, c), a[c]);
  }
  __syncwarp();                            // lanes i and i + 16 read the same row
  if (lane < 16) {
#pragma unroll
    for (int c = 0; c < 16; ++c)
      if (c <= i) sA[(j0 + i) * LD + j0 + c] = a[c];
    s_inv[j0 + i] = myinv;
  }
}

// Solves the Kd x Kd system (Kd = 16 * panels) whose lower triangle is rows 0 .. Kd-1 of sA and
// whose right-hand side is row Kd; the solution replaces row Kd.  All NT threads, MB >= panels.
//
// Blocked right-looking Cholesky in panels of 16 columns with two barriers a panel.  The
// right-hand side travels as one more row, so the forward substitution comes with the
// factorisation; warp 5 updates and factors the next diagonal block while warps 0 to 3 update the
// rest of the trailing matrix and warp 4 the right-hand side.  What bounds it is that chain of
// dependent steps, hidden by the other CTAs of the SM.
template <int MB>
__device__ __forceinline__ void chol_solve(float* sA, int LD, float* s_inv, int panels, int tid) {
  const int lane = tid & 31, warp = tid >> 5;
  const int Kd = 16 * panels;
  if (warp == 5) diag_factor(sA, LD, s_inv, 0, lane);
  __syncthreads();
  for (int j0 = 0; j0 < Kd; j0 += 16) {
    const int j1 = j0 + 16, m = Kd - j1;
    if (tid <= m) {                        // L21 = A21 L11^-T, one row per thread, the last is b
      float* rowp = sA + (j1 + tid) * LD + j0;
      float x[16];
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        float v = rowp[c];
#pragma unroll
        for (int q = 0; q < c; ++q) v = fmaf(-x[q], sA[(j0 + c) * LD + j0 + q], v);
        x[c] = v * s_inv[j0 + c];
      }
#pragma unroll
      for (int c = 0; c < 16; ++c) rowp[c] = x[c];
    }
    __syncthreads();
    if (m == 0) break;
    if (warp < 4) {                        // A22 -= L21 L21^T below the diagonal, all but block (0, 0)
      // rows ty + 8 i, columns tx + 16 j: j <= i / 2
      constexpr int TB = MB > 1 ? MB - 1 : 1;
      const int tx = tid & 15, ty = tid >> 4, mb = m >> 4;
      float t[TB * (TB + 1)];
#pragma unroll
      for (int e = 0; e < TB * (TB + 1); ++e) t[e] = 0.f;
#pragma unroll 2
      for (int q = 0; q < 16; ++q) {
        float lc[TB];
#pragma unroll
        for (int i = 0; i < TB; ++i) lc[i] = i < mb ? sA[(j1 + tx + 16 * i) * LD + j0 + q] : 0.f;
#pragma unroll
        for (int i = 1; i < TB; ++i)
          if (i < mb) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const float lr = sA[(j1 + ty + 16 * i + 8 * h) * LD + j0 + q];
#pragma unroll
              for (int j = 0; j <= i; ++j) t[i * (i + 1) + 2 * j + h] = fmaf(lr, lc[j], t[i * (i + 1) + 2 * j + h]);
            }
          }
      }
#pragma unroll
      for (int i = 1; i < TB; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int r = j1 + ty + 16 * i + 8 * h, c = j1 + tx + 16 * j;
            if (i < mb && c <= r) sA[r * LD + c] -= t[i * (i + 1) + 2 * j + h];
          }
    } else if (warp == 4) {
      for (int c = lane; c < m; c += 32) {
        float v = sA[Kd * LD + j1 + c];
#pragma unroll
        for (int q = 0; q < 16; ++q) v = fmaf(-sA[Kd * LD + j0 + q], sA[(j1 + c) * LD + j0 + q], v);
        sA[Kd * LD + j1 + c] = v;
      }
    } else {
      const int r = j1 + (lane & 15), c0 = j1 + 8 * (lane >> 4);
      float v[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) v[c] = sA[r * LD + c0 + c];
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const float l = sA[r * LD + j0 + q];
#pragma unroll
        for (int c = 0; c < 8; ++c) v[c] = fmaf(-l, sA[(c0 + c) * LD + j0 + q], v[c]);
      }
#pragma unroll
      for (int c = 0; c < 8; ++c) sA[r * LD + c0 + c] = v[c];
      __syncwarp();
      diag_factor(sA, LD, s_inv, j1, lane);
    }
    __syncthreads();
  }
  // backward: L^T w = y, last panel first
  float* sb = sA + Kd * LD;
  for (int j0 = Kd - 16; j0 >= 0; j0 -= 16) {
    if (tid < 32) {
      float l[16];
#pragma unroll
      for (int c = 0; c < 16; ++c) l[c] = (lane < c) ? sA[(j0 + c) * LD + j0 + lane] : 0.f;
      const float inv = lane < 16 ? s_inv[j0 + lane] : 0.f;
      float bv = lane < 16 ? sb[j0 + lane] : 0.f;
#pragma unroll
      for (int c = 15; c >= 0; --c) {
        const float wc = __shfl_sync(0xffffffffu, bv * inv, c);
        if (lane == c) bv = wc;
        else bv = fmaf(-l[c], wc, bv);      // l[c] is zero from lane c on
      }
      if (lane < 16) sb[j0 + lane] = bv;
    }
    __syncthreads();
    if (tid < j0) {
      float v = sb[tid];
#pragma unroll
      for (int q = 0; q < 16; ++q) v = fmaf(-sA[(j0 + q) * LD + tid], sb[j0 + q], v);
      sb[tid] = v;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------- primal form
// 32 x 64 blocks of the lower triangle (32 x 32 at K = 32), one per warp; with fewer than six blocks
// several warps share one and split the rows.  A lane owns 8 x 8 values, so an item row costs it four
// 16-byte shared-memory loads for 64 multiply-adds.  A 16-byte load takes four passes of the shared
// memory however many lanes read the same word, and with 4 x 8 values per lane (ten 32 x 32 blocks)
// those passes were the bound: 77 % of all cycles, 174 cycles a rating against 167 here.
// Item rows arrive by asynchronous copies two stages ahead.
template <int K>
__global__ void __launch_bounds__(NT, 3) als_primal_kernel(AlsArgs a) {
  constexpr int LD = K + 1;
  constexpr int CW = K == 32 ? 1 : 2;                      // 16-byte pieces of columns per lane
  constexpr int NB = K == 32 ? 1 : (K == 64 ? 2 : 6), GR = 6 / NB;
  extern __shared__ __align__(16) float sm[];
  float* sA = sm;                       // (K + 1) x LD, under it three stages of RS x K item rows
  __shared__ float s_inv[K];
  __shared__ float s_r[3][RS];
  __shared__ int s_seg;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int panels = (a.k + 15) / 16, Kd = 16 * panels;
  const int blk = warp % NB, grp = warp / NB;
  const int bi = blk < 4 ? blk : blk - 2, bj = blk < 4 ? 0 : 1;   // (0..3, 0), (2..3, 1)
  const int row0 = 32 * bi + 8 * (lane >> 3), col0 = 64 * bj + 4 * (lane & 7);
  const int n_big = a.counters[C_BIG], n_seg = n_big + a.counters[C_SMALL];
  for (;;) {
    __syncthreads();                    // the previous system is done with shared memory
    if (tid == 0) s_seg = atomicAdd(a.counters + C_TICKET, 1);
    __syncthreads();
    const int t = s_seg;
    if (t >= n_seg) return;
    const int at = t < n_big ? t : a.seg_cap - 1 - (t - n_big);
    const int u = a.seg_user[at], slot = a.seg_slot[at];
    const long long p0 = a.user_ptr[u] + (long long)a.seg_piece[at] * a.piece;
    const long long left = a.user_ptr[u + 1] - p0;
    const int cnt = (int)(slot >= 0 && left > a.piece ? a.piece : left);
    const int ns = (cnt + RS - 1) / RS;
    if (a.k < K)                        // columns behind the rank stay zero in every stage
      for (int e = tid; e < 3 * RS * (K - a.k); e += NT) sm[(e / (K - a.k)) * K + a.k + e % (K - a.k)] = 0.f;
    u64 acc[8][2 * CW];                 // pairs of neighbouring columns
    float b1 = 0.f;                     // entry tid of H^T a
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 2 * CW; ++j) acc[i][j] = 0ull;
    int idx[4];                         // item rows of the warp's rows of the stage to come
    auto fetch_idx = [&](int s) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int r = s * RS + warp + 6 * q;
        idx[q] = r < cnt ? __ldg(a.item_idx + p0 + r) : -1;
      }
    };
    auto stage = [&](int s) {
      if (s < ns) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int r = warp + 6 * q;
          stage_row(sm + ((s % 3) * RS + r) * K, idx[q] >= 0 ? a.H + (long long)idx[q] * a.k : nullptr, a.H, a.k,
                    a.vec, lane);
          if (lane == 0)
            __pipeline_memcpy_async(&s_r[s % 3][r], idx[q] >= 0 ? a.rating + p0 + s * RS + r : a.rating, 4,
                                    idx[q] >= 0 ? 0 : 4);
        }
      }
      __pipeline_commit();
    };
    fetch_idx(0);
    stage(0);
    fetch_idx(1);
    stage(1);
    fetch_idx(2);
    for (int s = 0; s < ns; ++s) {
      __pipeline_wait_prior(1);
      __syncthreads();
      stage(s + 2);
      fetch_idx(s + 3);
      const float* sh = sm + (s % 3) * RS * K;
#pragma unroll 2
      for (int r = grp; r < RS; r += GR) {
        const float4 h0 = *reinterpret_cast<const float4*>(sh + r * K + row0);
        const float4 h1 = *reinterpret_cast<const float4*>(sh + r * K + row0 + 4);
        u64 x[2 * CW];
#pragma unroll
        for (int w = 0; w < CW; ++w) {
          const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(sh + r * K + col0 + 32 * w);
          x[2 * w] = v.x; x[2 * w + 1] = v.y;
        }
        const float h[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const u64 hh = pack2(h[i], h[i]);
#pragma unroll
          for (int j = 0; j < 2 * CW; ++j) acc[i][j] = fma2(hh, x[j], acc[i][j]);
        }
      }
      if (tid < K) {
#pragma unroll 8
        for (int r = 0; r < RS; ++r) b1 = fmaf(s_r[s % 3][r], sh[r * K + tid], b1);
      }
    }
    __pipeline_wait_prior(0);
    bool mine = true;                   // this warp's sums go into the matrix
    if (slot >= 0) {
      float* gA = a.scratch + (long long)slot * (K * K + K);
#pragma unroll
      for (int w = 0; w < CW; ++w) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float4 v;
          unpack2(acc[i][2 * w], v.x, v.y);
          unpack2(acc[i][2 * w + 1], v.z, v.w);
          pcl_red_add4(gA + (row0 + i) * K + col0 + 32 * w, v);
        }
      }
      if (tid < K) atomicAdd(gA + K * K + tid, b1);
      __threadfence();
      __syncthreads();
      if (tid == 0) {
        const int pieces = (int)((a.user_ptr[u + 1] - a.user_ptr[u] + a.piece - 1) / a.piece);
        s_seg = atomicAdd(a.slot_count + slot, 1) == pieces - 1;
      }
      __syncthreads();
      if (!s_seg) continue;
      __threadfence();
      mine = grp == 0;
      if (mine) {
#pragma unroll
        for (int w = 0; w < CW; ++w) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float4 v = __ldcg(reinterpret_cast<const float4*>(gA + (row0 + i) * K + col0 + 32 * w));
            acc[i][2 * w] = pack2(v.x, v.y);
            acc[i][2 * w + 1] = pack2(v.z, v.w);
          }
        }
      }
      if (tid < K) b1 = __ldcg(gA + K * K + tid);
    }
    __syncthreads();                    // everyone is done with the last stage
#pragma unroll 1
    for (int g = 0; g < GR; ++g) {      // warps that share a block add one after the other
      if (grp == g && mine) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int w = 0; w < CW; ++w) {
            float v[4];
            unpack2(acc[i][2 * w], v[0], v[1]);
            unpack2(acc[i][2 * w + 1], v[2], v[3]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int r = row0 + i, c = col0 + 32 * w + j;
              if (c > r) continue;      // a block reaches past the diagonal: its other half is not needed
              if (g == 0) sA[r * LD + c] = v[j] + (r == c ? a.lambda : 0.f);
              else sA[r * LD + c] += v[j];
            }
          }
      }
      __syncthreads();
    }
    if (tid < Kd) sA[Kd * LD + tid] = b1;
    __syncthreads();
    chol_solve<K / 16>(sA, LD, s_inv, panels, tid);
    if (tid < a.k) a.W[(long long)u * a.k + tid] = sA[Kd * LD + tid];
  }
}

// --------------------------------------------------------------------- dual form, CTA per user
template <int NB2>                      // n <= 32 * NB2
__global__ void __launch_bounds__(NT, 3) als_dual_kernel(AlsArgs a, int cls) {
  constexpr int N = 32 * NB2, LD = N + 1, NB = NB2 * (NB2 + 1) / 2, GR = 6 / NB;   // three or six 32 x 32 blocks
  extern __shared__ __align__(16) float sm[];
  const int KS = (a.k + 31) / 32 * 32 + 4;         // row pitch: eight rows four banks apart
  float* sh = sm;                       // N x KS item rows
  float* sA = sm + N * KS;              // (N + 1) x LD
  __shared__ float s_inv[N];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int blk = warp % NB, grp = warp / NB;
  int bi = 0;
  while ((bi + 1) * (bi + 2) / 2 <= blk) ++bi;
  const int bj = blk - bi * (bi + 1) / 2;
  const int row0 = 32 * bi + (lane >> 2), col0 = 32 * bj + (lane & 3);
  const int n_list = a.counters[C_T16 + cls], k4 = (a.k + 3) / 4;
  const int* list = a.user_list + cls * a.n_users;
  // zeros behind the rank, and finite values in rows no user has filled yet
  for (int e = tid; e < N * KS; e += NT) sh[e] = 0.f;
  for (int at = blockIdx.x; at < n_list; at += gridDim.x) {
    const int u = list[at];
    const long long p0 = a.user_ptr[u];
    const int n = (int)(a.user_ptr[u + 1] - p0), panels = (n + 15) / 16, Kd = 16 * panels;
    __syncthreads();
    for (int r = warp; r < n; r += NT / 32)
      stage_row(sh + r * KS, a.H + (long long)__ldg(a.item_idx + p0 + r) * a.k, a.H, a.k, a.vec, lane);
    __pipeline_commit();
    __pipeline_wait_prior(0);
    __syncthreads();
    float acc[4][8];
    {
      u64 acc2[4][8];                   // sums over even and odd components
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc2[i][j] = 0ull;
#pragma unroll 1
      for (int c = grp; c < k4; c += GR) {
        ulonglong2 x[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const ulonglong2*>(sh + (row0 + 8 * i) * KS + 4 * c);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(sh + (col0 + 4 * j) * KS + 4 * c);
#pragma unroll
          for (int i = 0; i < 4; ++i) acc2[i][j] = fma2(x[i].y, y.y, fma2(x[i].x, y.x, acc2[i][j]));
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float e, o;
          unpack2(acc2[i][j], e, o);
          acc[i][j] = e + o;
        }
    }
#pragma unroll 1
    for (int g = 0; g < GR; ++g) {
      if (grp == g) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int r = row0 + 8 * i, c = col0 + 4 * j;
            // rows from n on: the unit matrix
            const float v = r < n && c < n ? acc[i][j] : 0.f;
            if (g == 0) sA[r * LD + c] = v + (r == c ? (r < n ? a.lambda : 1.f) : 0.f);
            else sA[r * LD + c] += v;
          }
      }
      __syncthreads();
    }
    if (tid < Kd) sA[Kd * LD + tid] = tid < n ? __ldg(a.rating + p0 + tid) : 0.f;
    __syncthreads();
    chol_solve<2 * NB2>(sA, LD, s_inv, panels, tid);
    if (tid < a.k) {                    // w = H_u^T y
      const float* y = sA + Kd * LD;
      float s0 = 0.f, s1 = 0.f;
      int i = 0;
      for (; i + 1 < n; i += 2) {
        s0 = fmaf(y[i], sh[i * KS + tid], s0);
        s1 = fmaf(y[i + 1], sh[(i + 1) * KS + tid], s1);
      }
      if (i < n) s0 = fmaf(y[i], sh[i * KS + tid], s0);
      a.W[(long long)u * a.k + tid] = s0 + s1;
    }
  }
}

// -------------------------------------------------------------------- dual form, warp per user
// n <= N (16 or 32).  Item rows in shared memory, the n x n matrix one row per lane in registers.
template <int N>
__global__ void __launch_bounds__(128) als_warp_kernel(AlsArgs a, int cls) {
  extern __shared__ __align__(16) float sm[];
  const int KS = (a.k + 31) / 32 * 32 + 4;
  constexpr int LG = N + 1, RI = N / 8, CJ = N / 4;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  float* sh = sm + wib * (N * KS + N * LG);
  float* sG = sh + N * KS;
  const int n_list = a.counters[C_T16 + cls], k4 = (a.k + 3) / 4;
  const int* list = a.user_list + cls * a.n_users;
  const int me = lane % N;
  for (int e = lane; e < N * KS; e += 32) sh[e] = 0.f;
  for (int at = blockIdx.x * 4 + wib; at < n_list; at += gridDim.x * 4) {
    const int u = list[at];
    const long long p0 = a.user_ptr[u];
    const int n = (int)(a.user_ptr[u + 1] - p0);
    const int idx = lane < n ? __ldg(a.item_idx + p0 + lane) : 0;
    float b = lane < n ? __ldg(a.rating + p0 + lane) : 0.f;
    __syncwarp();                       // the previous user's rows have been read
    for (int r = 0; r < n; ++r)
      stage_row(sh + r * KS, a.H + (long long)__shfl_sync(0xffffffffu, idx, r) * a.k, a.H, a.k, a.vec, lane);
    __pipeline_commit();
    __pipeline_wait_prior(0);
    __syncwarp();
    u64 acc[RI][CJ];                    // sums over even and odd components
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
      for (int j = 0; j < CJ; ++j) acc[i][j] = 0ull;
    const int r0 = lane >> 2, c0 = lane & 3;
#pragma unroll 1
    for (int c = 0; c < k4; ++c) {
      ulonglong2 x[RI];
#pragma unroll
      for (int i = 0; i < RI; ++i) x[i] = *reinterpret_cast<const ulonglong2*>(sh + (r0 + 8 * i) * KS + 4 * c);
#pragma unroll
      for (int j = 0; j < CJ; ++j) {
        const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(sh + (c0 + 4 * j) * KS + 4 * c);
#pragma unroll
        for (int i = 0; i < RI; ++i) acc[i][j] = fma2(x[i].y, y.y, fma2(x[i].x, y.x, acc[i][j]));
      }
    }
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
      for (int j = 0; j < CJ; ++j) {
        const int r = r0 + 8 * i, c = c0 + 4 * j;
        float e, o;
        unpack2(acc[i][j], e, o);
        sG[r * LG + c] = e + o + (r == c ? a.lambda : 0.f);
      }
    __syncwarp();
    float g[N];
#pragma unroll
    for (int c = 0; c < N; ++c) g[c] = sG[me * LG + c];
    __syncwarp();
    // Cholesky by columns, the right-hand side eliminated along; entries of rows and columns from n
    // on are leftovers that no lane below n reads
    float inv_me = 0.f;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      if (j < n) {
        const float d = sqrtf(fmaxf(__shfl_sync(0xffffffffu, g[j], j), 1e-30f));
        const float inv = 1.f / d;
        const float l = g[j] * inv;
        if (me == j) inv_me = inv;
        const float y = __shfl_sync(0xffffffffu, b, j) * inv;
        if (me == j) b = y;
        else if (me > j) b = fmaf(-l, y, b);
#pragma unroll
        for (int c = j + 1; c < N; ++c) g[c] = fmaf(-l, __shfl_sync(0xffffffffu, l, c), g[c]);
        if (lane < N) sG[me * LG + j] = l;
      }
    }
    __syncwarp();
#pragma unroll 1
    for (int j = n - 1; j >= 0; --j) {
      const float x = __shfl_sync(0xffffffffu, b * inv_me, j);
      if (me == j) b = x;
      else if (me < j) b = fmaf(-sG[j * LG + me], x, b);
    }
    // w = H_u^T y
    if (a.vec) {
      float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int i = 0; i < n; ++i) {
        const float y = __shfl_sync(0xffffffffu, b, i);
        if (4 * lane < a.k) {
          const float4 h = *reinterpret_cast<const float4*>(sh + i * KS + 4 * lane);
          w.x = fmaf(y, h.x, w.x); w.y = fmaf(y, h.y, w.y);
          w.z = fmaf(y, h.z, w.z); w.w = fmaf(y, h.w, w.w);
        }
      }
      if (4 * lane < a.k) {
        float* o = a.W + (long long)u * a.k + 4 * lane;
        o[0] = w.x; o[1] = w.y; o[2] = w.z; o[3] = w.w;
      }
    } else {
      float w[4] = {0.f, 0.f, 0.f, 0.f};
      for (int i = 0; i < n; ++i) {
        const float y = __shfl_sync(0xffffffffu, b, i);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (lane + 32 * q < a.k) w[q] = fmaf(y, sh[i * KS + lane + 32 * q], w[q]);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (lane + 32 * q < a.k) a.W[(long long)u * a.k + lane + 32 * q] = w[q];
    }
  }
}

// Largest resident grid of a persistent kernel with `smem` bytes, at most `need` blocks.
template <typename F>
int resident_grid(F kernel, int threads, size_t smem, long long need, int* grid) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
  if (e != cudaSuccess) return (int)e;
  const long long g = 148LL * (per_sm > 0 ? per_sm : 1);
  *grid = (int)(need < g ? need : g);
  return 0;
}

template <int K>
int launch_primal(const AlsArgs& a, long long max_seg, cudaStream_t stream) {
  size_t smem = (size_t)(K + 1) * (K + 1) * sizeof(float);
  if (smem < (size_t)3 * RS * K * sizeof(float)) smem = (size_t)3 * RS * K * sizeof(float);
  int grid = 0;
  const int rc = resident_grid(als_primal_kernel<K>, NT, smem, max_seg, &grid);
  if (rc != 0) return rc;
  als_clear_kernel<<<148 * 4, 256, 0, stream>>>(a.scratch, a.counters, K * K + K);
  als_primal_kernel<K><<<grid, NT, smem, stream>>>(a);
  return pcl_last_error();
}

template <int NB2>
int launch_dual(const AlsArgs& a, int cls, cudaStream_t stream) {
  constexpr int N = 32 * NB2;
  const int KS = (a.k + 31) / 32 * 32 + 4;
  const size_t smem = ((size_t)N * KS + (size_t)(N + 1) * (N + 1)) * sizeof(float);
  int grid = 0;
  const int rc = resident_grid(als_dual_kernel<NB2>, NT, smem, a.n_users, &grid);
  if (rc != 0) return rc;
  als_dual_kernel<NB2><<<grid, NT, smem, stream>>>(a, cls);
  return pcl_last_error();
}

template <int N>
int launch_warp(const AlsArgs& a, int cls, cudaStream_t stream) {
  const int KS = (a.k + 31) / 32 * 32 + 4;
  const size_t smem = 4 * ((size_t)N * KS + N * (N + 1)) * sizeof(float);
  int grid = 0;
  const int rc = resident_grid(als_warp_kernel<N>, 128, smem, (a.n_users + 3) / 4, &grid);
  if (rc != 0) return rc;
  als_warp_kernel<N><<<grid, 128, smem, stream>>>(a, cls);
  return pcl_last_error();
}

}  // namespace

// k <= 128, n_users < 2^31.  `nnz` is the length of item_idx / rating (user_ptr is ascending within
// [0, nnz]).  Users with more than `split` ratings are cut into pieces of `piece`.  Workspaces:
// scratch holds as many slots of K*K + K floats (K = k rounded up to 32 / 64 / 128, 16-byte aligned) as
// users are split (nnz / split at most) and slot_count as many ints; counters 8 ints; seg 3 x seg_cap ints
// with seg_cap >= n_users + nnz / piece + slots; user_list 4 x n_users ints.  Rows of W of users without
// ratings are not written.
PCL_API int pcl_als_solve(const long long* user_ptr, const int* item_idx, const float* rating, const float* H,
                          float* W, float* scratch, int* slot_count, int* counters, int* seg, int* user_list,
                          long long n_users, long long split, int piece, int seg_cap, int k, float lambda,
                          cudaStream_t stream) {
  if (n_users <= 0) return 0;
  if (k <= 0 || k > 128 || split <= 0 || piece <= 0 || n_users > 0x7fffffffLL) return (int)cudaErrorInvalidValue;
  const int vec = (k & 3) == 0 && (reinterpret_cast<uintptr_t>(H) & 15) == 0;
  AlsArgs a{user_ptr, item_idx, rating, H, W, scratch, slot_count, counters, seg, seg + seg_cap, seg + 2LL * seg_cap,
            user_list, n_users, split, piece, seg_cap, k, lambda, vec};
  cudaError_t e = cudaMemsetAsync(counters, 0, C_N * sizeof(int), stream);
  if (e != cudaSuccess) return (int)e;
  als_plan_kernel<<<(int)((n_users + 255) / 256), 256, 0, stream>>>(a);
  int rc = pcl_last_error();
  if (rc != 0) return rc;
  if (k <= 32) rc = launch_primal<32>(a, seg_cap, stream);
  else if (k <= 64) rc = launch_primal<64>(a, seg_cap, stream);
  else rc = launch_primal<128>(a, seg_cap, stream);
  if (rc != 0 || !(lambda > 0.f)) return rc;
  if (k > 64 && (rc = launch_dual<3>(a, 3, stream)) != 0) return rc;
  if (k > 33 && (rc = launch_dual<2>(a, 2, stream)) != 0) return rc;
  if (k > 17 && (rc = launch_warp<32>(a, 1, stream)) != 0) return rc;
  return k > 1 ? launch_warp<16>(a, 0, stream) : 0;
}
