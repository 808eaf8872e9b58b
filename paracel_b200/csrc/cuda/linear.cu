// Gradient kernels of the linear models (logistic regression, ridge, sparse
// L1-regularised logistic regression / Lasso).
//
// Math (reference: alg/classification/logistic_regression/lr.cpp:69-72, 119-145;
// alg/regression/ridge/ridge.hpp:73-96; tool/lr_l1_serial.cpp:46-73 for the L1
// objective): residual r = y - h(theta.x) with h = sigmoid (logistic) or identity
// (ridge), gradient accumulator g = sum_rows r * x, loss = log-loss or squared error.
// The accumulated g is what the reference's "dgd" method pushes with one bupdate per
// round; here it is written straight into the delta vector that dense_bupdate reduces.
//
// Dense kernel: a warp per row (or a few rows), per-block partial gradient, then a second
// kernel adds the blocks x d partials up in a fixed order, so that the result does not
// depend on atomics between blocks.
// Sparse kernel: CSR rows, one warp per row; features with index < hot_T (the most
// frequent ones after frequency renumbering) accumulate in shared memory per block,
// the others go to global memory with red.add.
#include <stdio.h>

#include "common.cuh"
#include <mutex>
#include "pcl_noalloc.h"

namespace {

struct DenseGradArgs {
  const float* X;      // n x d row-major
  const float* y;      // n
  const float* theta;  // d
  long long n;
  int d;
  int logistic;
  float* scratch;      // gridDim.x * d partial gradients + gridDim.x loss partials (as 2 floats each)
  int private_acc;     // 1: every warp owns a d-float accumulator in shared memory (no atomics)
};

__device__ __forceinline__ float sigmoidf_(float z) { return 1.f / (1.f + __expf(-z)); }

// residual of a row from its margin z; adds the row's loss
__device__ __forceinline__ float dg_residual(const DenseGradArgs& a, float z, float yy, double& loss) {
  if (a.logistic) {
    const float h = sigmoidf_(z);
    // log-loss with clamping so that a saturated sigmoid does not give inf
    const float hc = fminf(fmaxf(h, 1e-7f), 1.f - 1e-7f);
    loss += (yy == 1.f) ? -(double)__logf(hc) : -(double)__logf(1.f - hc);
    return yy - h;
  }
  const float r = yy - z;
  loss += (double)r * (double)r;
  return r;
}

// The block's partial gradient (the slots of its warps in s_g) and loss into the scratch.
__device__ __forceinline__ void dg_store_partial(const DenseGradArgs& a, const float* s_g, int slots,
                                                 const double* s_loss) {
  const int wpb = blockDim.x >> 5;
  float* part = a.scratch + (long long)blockIdx.x * a.d;
  for (int j = threadIdx.x; j < a.d; j += blockDim.x) {
    float v = s_g[j];
    for (int w = 1; w < slots; ++w) v += s_g[(long long)w * a.d + j];
    part[j] = v;
  }
  if (threadIdx.x == 0) {
    double l = 0.0;
    for (int w = 0; w < wpb; ++w) l += s_loss[w];
    reinterpret_cast<double*>(a.scratch + (((long long)gridDim.x * a.d + 1) & ~1LL))[blockIdx.x] = l;
  }
}

constexpr int dg_blocks_per_sm(int P) { return P >= 4 ? 2 : 4; }

// Rows of up to 128 * P floats: theta, the rows and this warp's gradient sums stay in registers, and
// X is read exactly once.  A warp takes ROWS rows per step, all their loads in flight before the first
// is used.  VEC: rows start on 16-byte boundaries (d a multiple of 4) and a lane takes columns
// 128 t + 4 lane + q; otherwise 128 t + 32 q + lane.
template <int P, int ROWS, bool VEC>
__global__ void __launch_bounds__(256, dg_blocks_per_sm(P)) dense_grad_rows_kernel(DenseGradArgs a) {
  extern __shared__ float s_g[];      // 8 x d
  __shared__ double s_loss[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  auto col = [&](int t, int q) { return VEC ? 128 * t + 4 * lane + q : 128 * t + 32 * q + lane; };
  float th[P][4], gacc[P][4];
#pragma unroll
  for (int t = 0; t < P; ++t)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      th[t][q] = col(t, q) < a.d ? __ldg(a.theta + col(t, q)) : 0.f;
      gacc[t][q] = 0.f;
    }
  double loss = 0.0;
  const long long step = (long long)gridDim.x * wpb * ROWS;
  for (long long row = ((long long)blockIdx.x * wpb + warp) * ROWS; row < a.n; row += step) {
    float x[ROWS][P][4], z[ROWS], yy[ROWS];
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      const bool in = row + k < a.n;
      const float* xp = a.X + (row + k) * a.d;
#pragma unroll
      for (int t = 0; t < P; ++t) {
        if constexpr (VEC) {
          float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
          if (in && col(t, 0) < a.d) v = __ldg(reinterpret_cast<const float4*>(xp + col(t, 0)));
          x[k][t][0] = v.x; x[k][t][1] = v.y; x[k][t][2] = v.z; x[k][t][3] = v.w;
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q) x[k][t][q] = in && col(t, q) < a.d ? __ldg(xp + col(t, q)) : 0.f;
        }
      }
      yy[k] = in ? __ldg(a.y + row + k) : 0.f;
    }
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      z[k] = 0.f;
#pragma unroll
      for (int t = 0; t < P; ++t)
#pragma unroll
        for (int q = 0; q < 4; ++q) z[k] = fmaf(x[k][t][q], th[t][q], z[k]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int k = 0; k < ROWS; ++k) z[k] += __shfl_xor_sync(0xffffffffu, z[k], o);
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      if (row + k >= a.n) break;
      const float r = dg_residual(a, z[k], yy[k], loss);
#pragma unroll
      for (int t = 0; t < P; ++t)
#pragma unroll
        for (int q = 0; q < 4; ++q) gacc[t][q] = fmaf(r, x[k][t][q], gacc[t][q]);
    }
  }
#pragma unroll
  for (int t = 0; t < P; ++t)
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (col(t, q) < a.d) s_g[warp * a.d + col(t, q)] = gacc[t][q];
  if (lane == 0) s_loss[warp] = loss;  // identical in every lane of the warp
  __syncthreads();
  dg_store_partial(a, s_g, wpb, s_loss);
}

// Any d: the row is read twice (the second time from cache).
__global__ void __launch_bounds__(256) dense_grad_kernel(DenseGradArgs a) {
  extern __shared__ float sm[];
  float* s_theta = sm;          // d
  float* s_g = sm + a.d;        // d, or 8 x d with private accumulators
  __shared__ double s_loss[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  for (int j = threadIdx.x; j < a.d; j += blockDim.x) s_theta[j] = a.theta[j];
  for (int j = threadIdx.x; j < (a.private_acc ? wpb : 1) * a.d; j += blockDim.x) s_g[j] = 0.f;
  __syncthreads();
  double loss = 0.0;
  for (long long row = (long long)blockIdx.x * wpb + warp; row < a.n; row += (long long)gridDim.x * wpb) {
    const float* x = a.X + row * a.d;
    float z = 0.f;
#pragma unroll 8
    for (int j = lane; j < a.d; j += 32) z = fmaf(x[j], s_theta[j], z);
    z = pcl_warp_sum(z);
    const float r = dg_residual(a, z, a.y[row], loss);
    if (a.private_acc) {
      // entry j of this warp's accumulator is only ever touched by lane j % 32 of this warp
      float* gw = s_g + (long long)warp * a.d;
#pragma unroll 8
      for (int j = lane; j < a.d; j += 32) gw[j] = fmaf(r, x[j], gw[j]);
    } else {
      for (int j = lane; j < a.d; j += 32) atomicAdd(&s_g[j], r * x[j]);
    }
  }
  if (lane == 0) s_loss[warp] = loss;  // identical in every lane of the warp
  __syncthreads();
  dg_store_partial(a, s_g, a.private_acc ? wpb : 1, s_loss);
}

// g[d] and *loss from the `blocks` partials, in a fixed order.  A block owns 32 columns: warp w sums
// the partials w, w + 32, ..., eight in flight per lane; block 0 sums the losses as well.  (When the
// last block of the gradient kernel added the partials up one after the other, that chain was most of
// a step on a small table: 20,000 x 100, ten steps 877 -> 539 us.)
constexpr int DS_W = 32;

__global__ void __launch_bounds__(32 * DS_W) dense_grad_sum_kernel(const float* scratch, int blocks, int d, float* g,
                                                                   double* loss) {
  __shared__ float s_p[DS_W][33];
  __shared__ double s_l[DS_W];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int j = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (j < d) {
#pragma unroll 8
    for (int b = warp; b < blocks; b += DS_W) s += __ldg(scratch + (long long)b * d + j);
  }
  s_p[warp][lane] = s;
  if (blockIdx.x == 0) {
    const double* lp = reinterpret_cast<const double*>(scratch + (((long long)blocks * d + 1) & ~1LL));
    double l = 0.0;
    for (int b = threadIdx.x; b < blocks; b += 32 * DS_W) l += __ldg(lp + b);
    l = pcl_warp_sum_d(l);
    if (lane == 0) s_l[warp] = l;
  }
  __syncthreads();
  const int jt = blockIdx.x * 32 + warp;         // warp w finishes column w
  const float t = pcl_warp_sum(s_p[lane][warp]);
  if (lane == 0 && jt < d) g[jt] = t;
  if (blockIdx.x == 0 && warp == 0) {
    const double l = pcl_warp_sum_d(s_l[lane]);
    if (lane == 0) *loss = l;
  }
}

struct SparseGradArgs {
  const long long* row_ptr;  // n + 1
  const int* cols;
  const float* vals;         // null: all ones
  const float* y;
  const float* theta;        // full local copy
  long long n;
  int logistic;
  int hot_T;                 // feature ids < hot_T accumulate in shared memory
  float* g;                  // accumulated into (caller zeroes it)
  double* loss;              // accumulated into
};

// Hot features (ids below hot_T) accumulate per CTA in shared memory as 32-bit fixed point
// (2^-14 units, native integer atomics: a floating-point shared-memory atomic add is a
// compare-and-swap loop that retries under contention, and the hottest features are hit by
// most warps of a CTA at once).  |residual * value| <= a few units and a CTA adds at most a
// few hundred thousand terms per feature, so 17 integer bits are ample.
constexpr float SG_FX = 16384.f, SG_FXI = 1.f / 16384.f;
#ifndef SG_ROWS_N
#define SG_ROWS_N 4
#endif
constexpr int SG_ROWS = SG_ROWS_N;
constexpr int SG_LONG = 4;

// residual of one row from its margin z; adds the row's loss
__device__ __forceinline__ float sg_residual(const SparseGradArgs& a, float z, float yy, double& loss) {
  if (a.logistic) {
    const float h = sigmoidf_(z);
    const float hc = fminf(fmaxf(h, 1e-7f), 1.f - 1e-7f);
    loss += (yy == 1.f) ? -(double)__logf(hc) : -(double)__logf(1.f - hc);
    return yy - h;
  }
  const float r = yy - z;
  loss += (double)r * (double)r;
  return r;
}

// FX: fixed point.  Squared-loss residuals are unbounded and keep floating-point sums (in shared memory
// too: sent straight to global memory, the additions to the hottest features queued up at a few
// addresses and took six times as long as everything else).
template <bool FX>
__device__ __forceinline__ void sg_scatter(const SparseGradArgs& a, int* s_hot, int c, float t) {
  if (!FX && c < a.hot_T) atomicAdd(reinterpret_cast<float*>(s_hot) + c, t);
  else if (FX && c < a.hot_T && fabsf(t) < 64.f) atomicAdd(&s_hot[c], __float2int_rn(t * SG_FX));
  else atomicAdd(a.g + c, t);
}

// A warp takes SG_ROWS rows per step.  A row is a chain of dependent long-latency accesses (row
// pointers, column ids, gather of theta, then the atomics), and with one row per warp the SM had
// only as many chains in flight as resident warps (long scoreboard 17 stall cycles per issue).
// Rows of up to 64 non-zeros keep their ids and values in registers between the margin and the
// scatter.  If a step has a longer row, its rows are taken one after the other, 32 SG_LONG entries in
// flight at a time (rows of up to that many keep them in registers too).
// Measured on 50 M x 2^24 with 40 non-zeros per row: 1 / 2 / 4 / 8 rows per step gave 2.04 / 3.16 /
// 3.36 / 2.06 G samples/s (eight rows cost too many registers).  The stream (limits, ids, values) of short
// rows is read one step ahead and past the caches' stock of weights: 2 M such rows 540 -> 412 us, with
// values 561 -> 426 us, against all of it read in its own step.
// Long rows as a loop over 32 entries, and their steps' registers filled for nothing: 2 M rows of 80 entries
// 1350 us, 1 M of 90 with values 620 us; SG_LONG 2 / 3 / 4 / 6: 1061 / 817 / 832 / 866 and 498 / 371 / 385 /
// 412 us, rows of 300 entries 354 / 311 / 291 / 307 us.
template <bool VALS, bool FX>
__global__ void __launch_bounds__(256, 4) sparse_grad_kernel(SparseGradArgs a) {
  extern __shared__ int s_hot[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  for (int j = threadIdx.x; j < a.hot_T; j += blockDim.x) s_hot[j] = 0;
  __syncthreads();
  double loss = 0.0;
  const long long stride = (long long)gridDim.x * wpb;
  // limits of a step's rows and, if all of them are short, their ids and values, read one step ahead
  bool shortrows = true;
  int c[2 * SG_ROWS];
  float v[VALS ? 2 * SG_ROWS : 1];
  long long nb[SG_ROWS], ne[SG_ROWS];
  auto limits = [&](long long row0) {
#pragma unroll
    for (int k = 0; k < SG_ROWS; ++k) {
      const long long row = row0 + k * stride;
      const bool has = row < a.n;
      nb[k] = has ? __ldg(a.row_ptr + row) : 0;
      ne[k] = has ? __ldg(a.row_ptr + row + 1) : 0;
    }
  };
  auto entries = [&]() {
    shortrows = true;
#pragma unroll
    for (int k = 0; k < SG_ROWS; ++k) shortrows &= ne[k] - nb[k] <= 64;
#pragma unroll
    for (int q = 0; q < 2 * SG_ROWS; ++q) {
      const long long p = nb[q >> 1] + (q & 1) * 32 + lane;
      const bool in = shortrows && p < ne[q >> 1];
      c[q] = in ? __ldcs(a.cols + p) : -1;
      if (VALS) v[VALS ? q : 0] = in ? __ldcs(a.vals + p) : 1.f;
    }
  };
  long long row0 = (long long)blockIdx.x * wpb + warp;
  if (row0 < a.n) {
    limits(row0);
    entries();
  }
  for (; row0 < a.n; row0 += SG_ROWS * stride) {
    const long long next = row0 + SG_ROWS * stride;
    if (shortrows) {
      limits(next);                              // rows past the end: empty
      float t[2 * SG_ROWS];
#pragma unroll
      for (int q = 0; q < 2 * SG_ROWS; ++q) t[q] = c[q] >= 0 ? __ldg(a.theta + c[q]) : 0.f;
      float yy[SG_ROWS];
#pragma unroll
      for (int k = 0; k < SG_ROWS; ++k) yy[k] = row0 + k * stride < a.n ? __ldcs(a.y + row0 + k * stride) : 0.f;
      int c0[2 * SG_ROWS];
      float v0[VALS ? 2 * SG_ROWS : 1];
#pragma unroll
      for (int q = 0; q < 2 * SG_ROWS; ++q) {
        c0[q] = c[q];
        if (VALS) v0[VALS ? q : 0] = v[VALS ? q : 0];
      }
      entries();
      float z[SG_ROWS];
#pragma unroll
      for (int k = 0; k < SG_ROWS; ++k)
        z[k] = VALS ? fmaf(v0[VALS ? 2 * k : 0], t[2 * k], v0[VALS ? 2 * k + 1 : 0] * t[2 * k + 1]) : t[2 * k] + t[2 * k + 1];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < SG_ROWS; ++k) z[k] += __shfl_xor_sync(0xffffffffu, z[k], o);
#pragma unroll
      for (int k = 0; k < SG_ROWS; ++k) {
        if (row0 + k * stride >= a.n) break;
        const float r = sg_residual(a, z[k], yy[k], loss);
        if (c0[2 * k] >= 0) sg_scatter<FX>(a, s_hot, c0[2 * k], VALS ? r * v0[VALS ? 2 * k : 0] : r);
        if (c0[2 * k + 1] >= 0) sg_scatter<FX>(a, s_hot, c0[2 * k + 1], VALS ? r * v0[VALS ? 2 * k + 1 : 0] : r);
      }
      continue;
    }
    // some row is long: lanes 2 k and 2 k + 1 hold the limits of row k of this step and of the next, which
    // leaves the registers to the loops
    auto lane_limit = [&](long long first) -> long long {
      const long long row = first + (lane >> 1) * stride;
      return lane < 2 * SG_ROWS && row < a.n ? __ldg(a.row_ptr + row + (lane & 1)) : 0;
    };
    const long long lim = lane_limit(row0), ahead = lane_limit(next);
#pragma unroll 1
    for (int k = 0; k < SG_ROWS; ++k) {
      const long long row = row0 + k * stride;
      if (row >= a.n) break;
      const long long b = __shfl_sync(0xffffffffu, lim, 2 * k), e = __shfl_sync(0xffffffffu, lim, 2 * k + 1);
      const float y1 = __ldg(a.y + row);
      int cl[SG_LONG];
      float vl[SG_LONG];
      auto fetch = [&](long long q) {              // the row's entries q .. q + 32 SG_LONG - 1, all loads in flight
#pragma unroll
        for (int j = 0; j < SG_LONG; ++j) {
          const long long p = q + 32 * j + lane;
          cl[j] = p < e ? __ldg(a.cols + p) : -1;
          vl[j] = VALS && p < e ? __ldg(a.vals + p) : 1.f;
        }
      };
      float zz = 0.f;
#pragma unroll 1
      for (long long q = b; q < e; q += 32 * SG_LONG) {
        fetch(q);
#pragma unroll
        for (int j = 0; j < SG_LONG; ++j)
          if (cl[j] >= 0) zz = fmaf(vl[j], __ldg(a.theta + cl[j]), zz);
      }
      zz = pcl_warp_sum(zz);
      const float r = sg_residual(a, zz, y1, loss);
#pragma unroll 1
      for (long long q = b; q < e; q += 32 * SG_LONG) {
        if (e - b > 32 * SG_LONG) fetch(q);        // else they are still there
#pragma unroll
        for (int j = 0; j < SG_LONG; ++j)
          if (cl[j] >= 0) sg_scatter<FX>(a, s_hot, cl[j], r * vl[j]);
      }
    }
#pragma unroll
    for (int k = 0; k < SG_ROWS; ++k) {
      nb[k] = __shfl_sync(0xffffffffu, ahead, 2 * k);
      ne[k] = __shfl_sync(0xffffffffu, ahead, 2 * k + 1);
    }
    entries();
  }
  __syncthreads();
  for (int j = threadIdx.x; j < a.hot_T; j += blockDim.x) {
    const float v = FX ? (float)s_hot[j] * SG_FXI : __int_as_float(s_hot[j]);
    if (v != 0.f) atomicAdd(a.g + j, v);
  }
  if (lane == 0 && loss != 0.0) atomicAdd(a.loss, loss);
}

template <typename F>
int dg_launch(F kernel, const DenseGradArgs& a, int blocks, size_t smem, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  kernel<<<blocks, 256, smem, stream>>>(a);
  return pcl_last_error();
}

// The grid: one wave, and at least two steps a warp, since every block costs a row of partials.
template <int P, int ROWS>
int dg_launch_rows(const DenseGradArgs& a, int* blocks, cudaStream_t stream) {
  const long long most = 148LL * dg_blocks_per_sm(P), need = (a.n + 16 * ROWS - 1) / (16 * ROWS);
  if (*blocks > most) *blocks = (int)most;
  if (*blocks > need) *blocks = (int)need;
  const size_t smem = 8 * (size_t)a.d * sizeof(float);
  if ((a.d & 3) == 0 && (reinterpret_cast<uintptr_t>(a.X) & 15) == 0)
    return dg_launch(dense_grad_rows_kernel<P, ROWS, true>, a, *blocks, smem, stream);
  return dg_launch(dense_grad_rows_kernel<P, ROWS, false>, a, *blocks, smem, stream);
}

// Rows of up to 1024 floats are kept in registers; ROWS puts 16 values per lane in flight (32 from
// d > 256 on, where fewer warps are resident).
int launch_dense_grad(DenseGradArgs a, int blocks, float* g, double* loss, cudaStream_t stream) {
  // per-warp accumulators (8 warps) when they fit into shared memory, else one shared accumulator
  a.private_acc = (9 * (size_t)a.d * sizeof(float) <= 200 * 1024) ? 1 : 0;
  int rc;
  if (a.d <= 128) rc = dg_launch_rows<1, 4>(a, &blocks, stream);
  else if (a.d <= 256) rc = dg_launch_rows<2, 2>(a, &blocks, stream);
  else if (a.d <= 512) rc = dg_launch_rows<4, 2>(a, &blocks, stream);
  else if (a.d <= 1024) rc = dg_launch_rows<8, 1>(a, &blocks, stream);
  else rc = dg_launch(dense_grad_kernel, a, blocks, (a.private_acc ? 9 : 2) * (size_t)a.d * sizeof(float), stream);
  if (rc != 0) return rc;
  dense_grad_sum_kernel<<<(a.d + 31) / 32, 32 * DS_W, 0, stream>>>(a.scratch, blocks, a.d, g, loss);
  return pcl_last_error();
}

}  // namespace

// Number of floats of scratch the dense gradient needs for `blocks` blocks and dimension d.
PCL_API long long pcl_lr_dense_scratch_floats(int blocks, int d) {
  return (long long)blocks * d + 2LL * blocks + 4;
}

// g[d] = sum_rows (y - h(theta.x)) x, *loss = summed loss.  `scratch` must hold
// pcl_lr_dense_scratch_floats(blocks, d) floats (8-byte aligned).  d <= 12000.
PCL_API int pcl_lr_dense_grad(const float* X, const float* y, const float* theta, long long n, int d,
                              int logistic, float* g, double* loss, float* scratch, int blocks,
                              cudaStream_t stream) {
  if (n <= 0 || d <= 0) return (int)cudaErrorInvalidValue;
  if (d > 12000) return (int)cudaErrorInvalidValue;
  if (blocks <= 0) blocks = 148 * 2;
  long long need = (n + 7) / 8;
  if (need < blocks) blocks = (int)need;
  DenseGradArgs a{X, y, theta, n, d, logistic, scratch, 0};
  return launch_dense_grad(a, blocks, g, loss, stream);
}

PCL_API int pcl_lr_sparse_grad(const long long* row_ptr, const int* cols, const float* vals,
                               const float* y, const float* theta, long long n, int logistic,
                               int hot_T, float* g, double* loss, int blocks, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (hot_T < 0 || hot_T > 24 * 1024) return (int)cudaErrorInvalidValue;
  SparseGradArgs a{row_ptr, cols, vals, y, theta, n, logistic, hot_T, g, loss};
  size_t smem = (size_t)hot_T * sizeof(float);
  auto kernel = vals != nullptr ? (logistic ? sparse_grad_kernel<true, true> : sparse_grad_kernel<true, false>)
                                : (logistic ? sparse_grad_kernel<false, true> : sparse_grad_kernel<false, false>);
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return (int)e;
  if (blocks <= 0) {
    // as many blocks as are resident at once (the kernel is bound by gather / atomic latency,
    // so every resident warp counts; the shared-memory table of hot features sets the limit)
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, smem);
    if (e != cudaSuccess) return (int)e;
    blocks = 148 * (per_sm > 0 ? per_sm : 4);
  }
  long long need = (n + 7) / 8;
  if (need < blocks) blocks = (int)need;
  kernel<<<blocks, 256, smem, stream>>>(a);
  return pcl_last_error();
}

// ---------------------------------------------------------------------------
// Allocation-free variant of the dense gradient (declared in pcl_noalloc.h).
//
// Some hosts of this library may not call cudaMalloc at all: a serving process
// that handed all of its HBM to one arena at start-up, a plug-in that runs
// inside somebody else's memory pool, or a latency-critical loop where the
// implicit device synchronisation of cudaMalloc/cudaFree is not acceptable.  For
// them the block partials live in the file-scope device array below instead of
// a caller-provided scratch tensor.  The price: every GPU that loads this library carries the
// PCL_NOALLOC_MAX_FLOATS * 4 bytes (4 MiB) until the process exits, and all
// calls on one device share the array, so two calls that overlap on the GPU
// (different streams) would overwrite each other's partials.
static __device__ __align__(256) float g_noalloc_scratch[PCL_NOALLOC_MAX_FLOATS];

namespace {
struct NoAllocSlot {
  float* scratch = nullptr;
  bool ready = false;
};
NoAllocSlot g_noalloc_slots[64];        // filled under g_noalloc_mutex, one entry per device
std::mutex g_noalloc_mutex;
thread_local char g_noalloc_msg[256] = "";   // last message of the calling host thread

int noalloc_fail(cudaError_t e, const char* what) {
  snprintf(g_noalloc_msg, sizeof(g_noalloc_msg), "pcl_lr_dense_grad_noalloc: %s failed: %s", what,
           cudaGetErrorString(e));
  return (int)e;
}
}  // namespace

PCL_API const char* pcl_lr_dense_grad_noalloc_error() { return g_noalloc_msg; }

PCL_API int pcl_lr_dense_grad_noalloc(const float* X, const float* y, const float* theta, long long n,
                                      int d, int logistic, float* g, double* loss, int blocks,
                                      cudaStream_t stream) {
  g_noalloc_msg[0] = 0;
  if (n <= 0 || d <= 0 || d > 12000) {
    snprintf(g_noalloc_msg, sizeof(g_noalloc_msg), "pcl_lr_dense_grad_noalloc: need n > 0 and 0 < d <= 12000 (got n=%lld d=%d)", n, d);
    return (int)cudaErrorInvalidValue;
  }
  if (blocks <= 0) blocks = 148 * 2;
  long long need_blocks = (n + 7) / 8;
  if (need_blocks < blocks) blocks = (int)need_blocks;
  const long long need = (long long)blocks * d + 2LL * blocks + 4;
  if (need > (long long)PCL_NOALLOC_MAX_FLOATS) {
    snprintf(g_noalloc_msg, sizeof(g_noalloc_msg),
             "pcl_lr_dense_grad_noalloc: %d blocks x d=%d needs %lld floats of scratch, the built-in "
             "array holds %d; use fewer blocks or pcl_lr_dense_grad with your own scratch",
             blocks, d, need, (int)PCL_NOALLOC_MAX_FLOATS);
    return (int)cudaErrorInvalidValue;
  }
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return noalloc_fail(e, "cudaGetDevice");
  if (dev < 0 || dev >= 64) {
    snprintf(g_noalloc_msg, sizeof(g_noalloc_msg), "pcl_lr_dense_grad_noalloc: device index %d not supported", dev);
    return (int)cudaErrorInvalidDevice;
  }
  NoAllocSlot& slot = g_noalloc_slots[dev];
  std::lock_guard<std::mutex> guard(g_noalloc_mutex);   // set-up and launch of one call at a time
  if (!slot.ready) {
    // One-time set-up for this device (it is the current device): translate the symbol
    // into a device address.  In host code the array name is only a stand-in.
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) {
      snprintf(g_noalloc_msg, sizeof(g_noalloc_msg), "cudaGetSymbolAddress(scratch) failed: %s", cudaGetErrorString(e));
      return (int)e;
    }
    slot.scratch = (float*)p;
    slot.ready = true;
  }
  // the partials are fully overwritten by the first kernel before the second reads them
  DenseGradArgs a{X, y, theta, n, d, logistic, slot.scratch, 0};
  const int rc = launch_dense_grad(a, blocks, g, loss, stream);
  if (rc != 0) return noalloc_fail((cudaError_t)rc, "kernel launch");
  return 0;
}
