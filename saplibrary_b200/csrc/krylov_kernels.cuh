// FP64 kernels of the Krylov loop: SpMV (banded row-major and CSR), BLAS-1
// updates and deterministic fused dot products.
#pragma once

#include <algorithm>

#include "common.cuh"

namespace sapb {

// y = A x for the row-major FP64 band of MVBanded (sap/spmv.h:27-74,
// sap/device/matrix_multiply.cuh:301-350): one warp per row, coalesced
// reads of the row's 2K+1 values.
static __global__ void __launch_bounds__(256)
k_spmv_banded(const double* __restrict__ A, const double* __restrict__ x, double* __restrict__ y, int n, int K) {
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  const long long SW = 2LL * K + 1;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
    const int lo = max(0, i - K), hi = min(n - 1, i + K);
    const double* row = A + (long long)i * SW + K - i;  // row[j] = A(i, j)
    double acc = 0.0;
    for (int j = lo + lane; j <= hi; j += 32) acc += row[j] * x[j];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (lane == 0) y[i] = acc;
  }
}

// The same for bands of at most kBandTile / 16 values per row: a CTA streams
// the contiguous entries of TR = 256 / LPR rows and the x they meet into shared
// memory (16 bytes per thread and load, all in flight together), then LPR
// threads per row add its products.  One warp per row, as above, leaves lanes
// idle below 32 values and keeps one row's loads in flight: 1,000,000 rows,
// K = 10: 110 us; 200,000 rows, K = 50: 55 us.  From 256 values per row on the
// warp is the better one (2,000,000 rows, K = 200: 6.0 TB/s).
constexpr int kBandTile = 4096;  // entries per CTA at most
constexpr int band_lanes(int SW) { return SW <= 16 ? 1 : SW <= 32 ? 2 : SW <= 64 ? 4 : SW <= 128 ? 8 : 16; }
template <int LPR>
static __global__ void __launch_bounds__(256)
k_spmv_band_tile(const double* __restrict__ A, const double* __restrict__ x, double* __restrict__ y, int n, int K) {
  constexpr int TR = 256 / LPR;
  extern __shared__ __align__(16) unsigned char band_raw[];
  const int SW = 2 * K + 1, r0 = blockIdx.x * TR, rows = min(TR, n - r0), t = threadIdx.x;
  double* sa = reinterpret_cast<double*>(band_raw);  // rows x SW
  double* xs = sa + TR * SW;                         // x[r0 - K ...]
  const double* src = A + (long long)r0 * SW;        // TR is even: 16-byte aligned
  const int cnt = rows * SW;
  for (int e = 2 * t; e + 1 < cnt; e += 512) cp_async16(sa + e, src + e);
  if ((cnt & 1) && t == 0) cp_async8(sa + cnt - 1, src + cnt - 1);
  cp_async_commit();
  for (int e = t; e < rows + 2 * K; e += 256) {
    const int c = r0 - K + e;
    xs[e] = c >= 0 && c < n ? x[c] : 0.0;
  }
  cp_async_wait<0>();
  __syncthreads();
  const int r = t / LPR, l = t % LPR, i = r0 + r;
  double acc = 0.0;
  if (r < rows) {
    const int k1 = min(2 * K, n - 1 - i + K);  // entries outside the matrix are not read
    for (int k = max(0, K - i) + l; k <= k1; k += LPR) acc += sa[r * SW + k] * xs[r + k];
  }
#pragma unroll
  for (int off = LPR / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (r < rows && l == 0) y[i] = acc;
}

// y = A x, FP64 CSR by row blocks (the product SpmvCusp delegates to,
// sap/spmv.h:110-121).  The rows are cut on the host into blocks of at most
// kSpmvRows rows and kSpmvNnz entries (csr_row_blocks); a row longer than
// kSpmvNnz is a block of its own.  A CTA streams its block's entries with
// fully coalesced loads of values and column indices, several per thread
// before their gathers of x, keeps the products in shared memory, then one
// thread per row adds its row's products in entry order.  A long row is
// summed by the whole CTA (strided partial sums, then a fixed-order
// reduction).
constexpr int kSpmvRows = 256;   // threads per CTA, rows per block at most
constexpr int kSpmvNnz = 2048;   // entries per block at most (16 KB of products)

static __global__ void __launch_bounds__(kSpmvRows)
k_spmv_csr_blocks(const int* __restrict__ blk, const int* __restrict__ rp, const int* __restrict__ ci,
                  const double* __restrict__ v, const double* __restrict__ x, double* __restrict__ y) {
  __shared__ double prod[kSpmvNnz];
  const int r0 = blk[blockIdx.x], r1 = blk[blockIdx.x + 1];
  const int e0 = rp[r0], cnt = rp[r1] - e0;
  const int t = threadIdx.x;
  if (cnt <= kSpmvNnz) {
    constexpr int U = kSpmvNnz / kSpmvRows;
    int c[U];
    double a[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int k = t + u * kSpmvRows;
      c[u] = k < cnt ? __ldg(ci + e0 + k) : 0;
      a[u] = k < cnt ? __ldg(v + e0 + k) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int k = t + u * kSpmvRows;
      if (k < cnt) prod[k] = a[u] * __ldg(x + c[u]);
    }
    __syncthreads();
    const int row = r0 + t;
    if (row < r1) {
      const int a0 = rp[row] - e0, a1 = rp[row + 1] - e0;
      double s = 0.0;
      for (int k = a0; k < a1; k++) s += prod[k];
      y[row] = s;
    }
  } else {  // one long row
    double s = 0.0;
    for (int k = t; k < cnt; k += kSpmvRows) s += __ldg(v + e0 + k) * __ldg(x + __ldg(ci + e0 + k));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if ((t & 31) == 0) prod[t >> 5] = s;
    __syncthreads();
    if (t == 0) {
      double tot = 0.0;
      for (int w = 0; w < kSpmvRows / 32; w++) tot += prod[w];
      y[r0] = tot;
    }
  }
}

// Row blocks of k_spmv_csr_blocks: boundaries b[0] = 0 < b[1] < ... = n, each
// block at most kSpmvRows rows and kSpmvNnz entries, or one longer row.
inline std::vector<int> csr_row_blocks(int n, const int* rp) {
  std::vector<int> b(1, 0);
  int r = 0;
  while (r < n) {
    const int r0 = r;
    while (r < n && r - r0 < kSpmvRows && rp[r + 1] - rp[r0] <= kSpmvNnz) r++;
    if (r == r0) r = r0 + 1;  // a row longer than kSpmvNnz
    b.push_back(r);
  }
  return b;
}

// z = a*x + b*y (cusp::blas::axpby)
static __global__ void k_axpby(int n, double a, const double* __restrict__ x, double b, const double* __restrict__ y,
                        double* __restrict__ z) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    z[i] = a * x[i] + b * y[i];
}
// y += a*x (cusp::blas::axpy)
static __global__ void k_axpy(int n, double a, const double* __restrict__ x, double* __restrict__ y) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] += a * x[i];
}
// z = b - y  (the true-residual recheck, axpby(b, APxx, rr0, 1, -1))
static __global__ void k_sub(int n, const double* __restrict__ b, const double* __restrict__ y, double* __restrict__ z) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) z[i] = b[i] - y[i];
}

// Up to 4 dot products sum_i x_q[i]*y_q[i] in one pass.  Block partials go to
// `part` (4 * gridDim.x doubles); the last block to finish reduces them, one
// warp per product, in a fixed order, so the result is deterministic for a
// given grid.  `counter` must be zero on entry and is zero again on exit.
// `out` may be page-locked host memory.
struct DotArgs {
  const double* x[4];
  const double* y[4];
  int nq;
};

constexpr int kDotBlocks = 296;
constexpr int kDotThreads = 512;
// blocks for vectors of length n: about four values per thread, two blocks per
// SM at most (n = 2,000: 1 block, whose sum needs no second stage's loads;
// with 296 blocks and a serial last sum the launch took 12 us at any n)
inline int dot_blocks(int n) { return std::max(1, std::min(kDotBlocks, (n + 4 * kDotThreads - 1) / (4 * kDotThreads))); }
// rows per thread of the size-proportional grid of the standalone dot entry point
constexpr int kDotItems = 16;
inline int dot_grid_for(long long n) {
  long long g = (n + (long long)kDotThreads * kDotItems - 1) / ((long long)kDotThreads * kDotItems);
  return (int)(g < 1 ? 1 : g);
}
static __device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}
// block sums of NQ accumulators, then (last block) of all blocks' partials
template <int NQ>
static __device__ __forceinline__ void dot_finish(const double* acc, int nq, double* part, unsigned int* counter,
                                                  double* out) {
  __shared__ double red[NQ][kDotThreads / 32];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    const double v = warp_sum(acc[q]);
    if (lane == 0) red[q][wid] = v;
  }
  __syncthreads();
  if (wid < NQ) {
    const double v = warp_sum(lane < kDotThreads / 32 ? red[wid][lane] : 0.0);
    if (lane == 0) {
      part[wid * gridDim.x + blockIdx.x] = v;
      __threadfence();
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (wid < nq) {
    double v = 0.0;
    for (int b = lane; b < (int)gridDim.x; b += 32) v += __ldcg(part + wid * gridDim.x + b);
    v = warp_sum(v);
    if (lane == 0) out[wid] = v;
  }
  if (threadIdx.x == 0) *counter = 0u;
}

static __global__ void __launch_bounds__(kDotThreads)
k_dots(int n, DotArgs a, double* __restrict__ part, unsigned int* __restrict__ counter,
       double* __restrict__ out) {
  double acc[4] = {0, 0, 0, 0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (q < a.nq) acc[q] += a.x[q][i] * a.y[q][i];
  }
  dot_finish<4>(acc, a.nq, part, counter, out);
}

// y += a x, then out[0] = y . y, in one pass: the update of the residual
// followed by its norm in BiCGStab(L).  Same grid, thread-to-row mapping and
// reduction order as k_dots, so out[0] equals k_dots(y, y) after k_axpy.
static __global__ void __launch_bounds__(kDotThreads)
k_axpy_sqnorm(int n, double a, const double* __restrict__ x, double* __restrict__ y, double* __restrict__ part,
              unsigned int* __restrict__ counter, double* __restrict__ out) {
  double acc = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double v = y[i] + a * x[i];
    y[i] = v;
    acc += v * v;
  }
  dot_finish<1>(&acc, 1, part, counter, out);
}

// Classical Gram-Schmidt of the Arnoldi step (flexible GMRES), one launch per
// pass instead of one dot and one axpy per basis vector:
//   k_mdot:  h[i] = V_i . w for i < m (blockIdx.y = i); block partials in
//            part[i][blockIdx.x], reduced in a fixed order by the last block of
//            each vector to finish (deterministic for a given grid), whose
//            counter returns to zero;
//   k_maxpy: w[r] -= h[0] V_0[r] + ... in order i = 0..m-1, one row per
//            thread (the basis pointers and h staged in shared memory).
constexpr int kMdotBlocks = 148;
constexpr int kMdotThreads = 256;
constexpr int kMaxBasis = 64;
// blocks per vector: about eight values per thread (64 blocks with a serial
// last sum: 14 us at 400,000 rows)
inline int mdot_blocks(int n) { return std::max(1, std::min(kMdotBlocks, (n + 8 * kMdotThreads - 1) / (8 * kMdotThreads))); }
static __global__ void __launch_bounds__(kMdotThreads)
k_mdot(int n, const double* const* __restrict__ vs, const double* __restrict__ w, double* __restrict__ part,
       unsigned int* __restrict__ ctr, double* __restrict__ h) {
  __shared__ double red[kMdotThreads / 32];
  __shared__ bool last;
  const int i = blockIdx.y, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const double* v = vs[i];
  double acc = 0.0;
#pragma unroll 4
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) acc += v[r] * w[r];
  acc = warp_sum(acc);
  if (lane == 0) red[wid] = acc;
  __syncthreads();
  if (wid == 0) {
    const double s = warp_sum(lane < kMdotThreads / 32 ? red[lane] : 0.0);
    if (lane == 0) {
      part[(size_t)i * gridDim.x + blockIdx.x] = s;
      __threadfence();
      last = atomicAdd(&ctr[i], 1u) == gridDim.x - 1;
    }
  }
  __syncthreads();
  if (last && wid == 0) {
    __threadfence();
    const double* pp = part + (size_t)i * gridDim.x;
    double s = 0.0;
    for (unsigned b = lane; b < gridDim.x; b += 32) s += __ldcg(pp + b);
    s = warp_sum(s);
    if (lane == 0) {
      h[i] = s;
      ctr[i] = 0u;
    }
  }
}

static __global__ void k_maxpy(int n, int m, const double* const* __restrict__ vs, const double* __restrict__ h,
                               double* __restrict__ w) {
  __shared__ const double* sv[kMaxBasis];
  __shared__ double sh[kMaxBasis];
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    sv[i] = vs[i];
    sh[i] = h[i];
  }
  __syncthreads();
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    double x = w[r];
    for (int i = 0; i < m; i++) x -= sh[i] * sv[i][r];
    w[r] = x;
  }
}

// w <- w / sqrt(nn[0]) when nn[0] > 0 (the Arnoldi normalisation, with the
// norm left on the device); block 0 also hands the step's 2 m coefficients
// (h1, h2) and nn to the host (page-locked: host[0..m), host[kMaxBasis ..),
// host[2 kMaxBasis]).
static __global__ void k_scale_inv_norm(int n, double* __restrict__ w, const double* __restrict__ nn, int m,
                                        const double* __restrict__ h1, const double* __restrict__ h2,
                                        double* __restrict__ host) {
  if (blockIdx.x == 0) {
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
      host[i] = h1[i];
      host[kMaxBasis + i] = h2[i];
    }
    if (threadIdx.x == 0) host[2 * kMaxBasis] = nn[0];
  }
  const double hn = sqrt(nn[0]);
  if (!(hn > 0)) return;
  const double a = 1.0 / hn;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) w[r] = a * w[r] + 0.0 * w[r];
}

// out = a x + b y + c z (cusp::blas::axpbypcz); out may alias an input
static __global__ void k_axpbypcz(int n, double a, const double* x, double b, const double* y, double c,
                                  const double* z, double* out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[i] = a * x[i] + b * y[i] + c * z[i];
}

}  // namespace sapb
