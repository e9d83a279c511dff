// Wide-band partitions (half-bandwidth of hundreds to thousands): every
// partition is treated as block tridiagonal with bs x bs blocks (bs >= K_p),
//     A_p = tridiag(F_{i-1}, D_i, E_i),
// and factored without pivoting blockwise:
//     D_i <- D_i - L_{i,i-1} U_{i-1,i};  D_i = L_ii U_ii;
//     U_{i,i+1} = L_ii^-1 E_i;  L_{i+1,i} = F_i U_ii^-1.
// These are exactly the L and U factors of the band LU (the LU without
// pivoting is unique), computed as dense block operations: the diagonal block
// LU is recursive and also returns L_ii^-1 and U_ii^-1, so every step except
// the leaves (one CTA each, see k_leaf) is a matrix product.  The apply
// then reduces to batched matrix-vector products per block row:
//     y_i = L_ii^-1 (f_i - L_{i,i-1} y_{i-1}),  x_i = U_ii^-1 (y_i - U_{i,i+1} x_{i+1}).
// Blocks are column-major (element (r, c) at c*bs + r); vectors are padded to
// nb*bs rows per partition, padding rows carry an identity diagonal.
#pragma once

#include <cooperative_groups.h>
#include <cuda_fp16.h>

#include <cstdlib>
#include <type_traits>

#include "precond_kernels.cuh"

namespace sapb {

// Granularity (rows) of the block sizes and of the recursion's splits.
constexpr int kLeaf = 32;

// COO entries of the diagonal blocks (row j, col l in band order) into the
// blocks of their partition: D (slot Dm), E = A_{i,i+1} (slot Em), F = A_{i+1,i} (slot Fm).
template <typename T>
__global__ void k_wb_scatter(const int* __restrict__ rows, const int* __restrict__ cols, const T* __restrict__ vals,
                             long long nz, const int* __restrict__ part_of_row, const int* __restrict__ pstart,
                             const int* __restrict__ psize, int bs, int nb, T* __restrict__ Dm, T* __restrict__ Em, T* __restrict__ Fm) {
  const long long BB = (long long)bs * bs;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nz;
       e += (long long)gridDim.x * blockDim.x) {
    const int j = rows[e], l = cols[e];
    const int p = part_of_row[j];
    const int a = j - pstart[p], c = l - pstart[p];
    if (c < 0 || c >= psize[p]) continue;  // outside the partition's diagonal block
    const int bi = a / bs, bj = c / bs;
    const long long off = (long long)(c - bj * bs) * bs + (a - bi * bs);
    if (bi == bj) Dm[((long long)p * nb + bi) * BB + off] = vals[e];
    else if (bj == bi + 1) Em[((long long)p * (nb - 1) + bi) * BB + off] = vals[e];
    else if (bj + 1 == bi) Fm[((long long)p * (nb - 1) + bj) * BB + off] = vals[e];
  }
}

// Identity diagonal on the padding rows [psize_p, nb*bs) of every partition.
template <typename T>
__global__ void k_wb_pad(T* __restrict__ Dm, const int* __restrict__ psize, int bs, int nb) {
  const int p = blockIdx.y;
  const long long BB = (long long)bs * bs;
  for (int r = psize[p] + blockIdx.x * blockDim.x + threadIdx.x; r < nb * bs; r += gridDim.x * blockDim.x) {
    const int bi = r / bs, q = r - bi * bs;
    Dm[((long long)p * nb + bi) * BB + (long long)q * bs + q] = T(1);
  }
}

// Band storage (column-major, 2K_p+1 rows per column, element (i, j) of a
// partition at boff + (j-start)*(2K_p+1) + K_p + (i-j)) into the blocks.
template <typename T>
__global__ void k_wb_from_band(const T* __restrict__ B, const long long* __restrict__ boff,
                               const int* __restrict__ kp, const int* __restrict__ psize, int bs, int nb,
                               T* __restrict__ Dm, T* __restrict__ Em, T* __restrict__ Fm) {
  const int p = blockIdx.y;
  const int Kp = kp[p], sz = psize[p];
  const long long SW = 2LL * Kp + 1, BB = (long long)bs * bs;
  const T* Bp = B + boff[p];
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < (long long)sz * SW;
       e += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(e / SW);
    const int a = c + (int)(e - (long long)c * SW) - Kp;
    if (a < 0 || a >= sz) continue;
    const T v = Bp[e];
    if (v == T(0)) continue;
    const int bi = a / bs, bj = c / bs;
    const long long off = (long long)(c - bj * bs) * bs + (a - bi * bs);
    if (bi == bj) Dm[((long long)p * nb + bi) * BB + off] = v;
    else if (bj == bi + 1) Em[((long long)p * (nb - 1) + bi) * BB + off] = v;
    else if (bj + 1 == bi) Fm[((long long)p * (nb - 1) + bj) * BB + off] = v;
  }
}

// Row-major FP64 band straight into the blocks (all of half-bandwidth K),
// scaled by sc_r sc_c (null: not scaled); grid (row tile of the partition,
// partition), 32 x 8 threads.  Saves the column-major band in between: 2M
// rows, K = 200 took 9.2 ms through it.
template <typename T>
__global__ void __launch_bounds__(256)
k_wb_from_rowmajor(const double* __restrict__ A, int K, const T* __restrict__ sc, const int* __restrict__ pstart,
                   const int* __restrict__ psize, int bs, int nb, T* __restrict__ Dm, T* __restrict__ Em,
                   T* __restrict__ Fm) {
  const int p = blockIdx.y, s = pstart[p], sz = psize[p], r0 = blockIdx.x * 32;
  if (r0 >= sz) return;
  const long long BB = (long long)bs * bs;
  band_transpose<T>(A, K, s + r0, s, s + sz, [&](int r, int c, T v) {
    if (r >= s + sz) return;
    if (sc) v *= sc[r] * sc[c];
    const int a = r - s, b = c - s, bi = a / bs, bj = b / bs;
    const long long off = (long long)(b - bj * bs) * bs + (a - bi * bs);
    if (bi == bj) Dm[((long long)p * nb + bi) * BB + off] = v;
    else if (bj > bi) Em[((long long)p * (nb - 1) + bi) * BB + off] = v;
    else Fm[((long long)p * (nb - 1) + bj) * BB + off] = v;
  });
}

// Batched copy of an m x n sub-matrix (column-major, leading dimensions lds/ldd).
template <typename T>
__global__ void k_sub_copy(const T* __restrict__ src, int lds, long long ss, T* __restrict__ dst, int ldd,
                           long long sd, int m, int n, T scale) {
  const int b = blockIdx.z;
  for (int c = blockIdx.y; c < n; c += gridDim.y)
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < m; r += gridDim.x * blockDim.x)
      dst[b * sd + (long long)c * ldd + r] = scale * src[b * ss + (long long)c * lds + r];
}

// Batched fill of an m x n sub-matrix with a value.
template <typename T>
__global__ void k_sub_fill(T* __restrict__ dst, int ldd, long long sd, int m, int n, T value) {
  const int b = blockIdx.z;
  for (int c = blockIdx.y; c < n; c += gridDim.y)
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < m; r += gridDim.x * blockDim.x)
      dst[b * sd + (long long)c * ldd + r] = value;
}

// Leaf of the recursive block LU: one CTA per batch element factors an n x n
// block (n <= leaf_max<T>) without pivoting (pivots boosted as in the band LU
// when `boost`, else a pivot below 1e-7 raises zero_flag) and writes L^-1
// (unit lower) to Li and U^-1 (upper) to Ui; M is only read.
//
// The whole block stays in shared memory (row-major, ld = n16 + 4), as 16 x 16
// tiles, one warp per tile and product:
//   * 16 pivots at a time: warp 0 factors the diagonal tile in registers; the
//     panels U12 = L^-1 A12 and L21 = A21 U^-1 follow by substitution, 32
//     columns or rows per warp, then A22 -= L21 U12, where warp 0 takes the
//     next diagonal tile and factors it at once while the other warps update
//     the rest and the last one inverts the tile's triangles in its place;
//   * the inverses of the two triangular factors grow by doubling, 16 -> 32 ->
//     64 -> 128: (L^-1)21 = -L22^-1 (L21 L11^-1), (U^-1)12 = -U11^-1 (U12
//     U22^-1), all pairs and both triangles at once, in place of L21 and U12.
// What bounds it is this chain of phases in one CTA per partition; larger
// leaves replace whole levels of the recursion, whose products cost a launch
// each (about 5 us, six on the chain of every level).  128 and 96 rows, 32
// partitions: 47 us, against some 120 us for 32-row leaves (12 us each) and the
// products of the two levels above them; 62 us with the inverses on the chain.
//
// tc: products between tiles of different 32-blocks run on the tensor cores
// in TF32 (mma.sync, FP32 accumulation), like the products of the recursion
// they stand for; within a 32-block, and without tc everywhere, they are FMAs
// in T.
template <typename T>
constexpr int leaf_max = sizeof(T) == 4 ? 128 : 96;  // two n x (n + 4) arrays of shared memory
constexpr int kLeafThreads = 512;
template <typename T>
inline size_t leaf_smem(int n) {
  const int n16 = (n + 15) / 16 * 16;
  return (size_t)2 * n16 * (n16 + 4) * sizeof(T);
}
enum { TILE_FULL = 0, TILE_UNIT_LOWER = 1, TILE_UPPER = 2 };
// element (r, c) of a 16 x 16 tile of G read as full, unit lower or upper
template <int TRI, typename T>
__device__ __forceinline__ T tile_el(const T* A, int ld, int r, int c) {
  const T v = A[r * ld + c];
  if constexpr (TRI == TILE_UNIT_LOWER) return r > c ? v : (r == c ? T(1) : T(0));
  if constexpr (TRI == TILE_UPPER) return r <= c ? v : T(0);
  return v;
}
__device__ __forceinline__ unsigned to_tf32(float v) {
  unsigned r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
  return r;
}
// acc += A B for 16 x 16 tiles, one warp.  Lane (g, t) = (lane / 4, lane % 4)
// holds rows g, g + 8 and columns 2t, 2t+1, 8+2t, 9+2t (the accumulator layout
// of mma.m16n8k8): acc[4 h + 2 i + j] = (g + 8 i, 8 h + 2 t + j).
template <int TA = TILE_FULL, int TB = TILE_FULL, typename T>
__device__ __forceinline__ void tile_mac(const T* A, const T* B, int ld, bool tc, T acc[8]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  if constexpr (sizeof(T) == 4) {
    if (tc) {
#pragma unroll
      for (int k = 0; k < 16; k += 8) {
        const unsigned a0 = to_tf32(tile_el<TA>(A, ld, g, k + t)), a1 = to_tf32(tile_el<TA>(A, ld, g + 8, k + t)),
                       a2 = to_tf32(tile_el<TA>(A, ld, g, k + t + 4)),
                       a3 = to_tf32(tile_el<TA>(A, ld, g + 8, k + t + 4));
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const unsigned b0 = to_tf32(tile_el<TB>(B, ld, k + t, 8 * h + g)),
                         b1 = to_tf32(tile_el<TB>(B, ld, k + t + 4, 8 * h + g));
          asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
              "{%0,%1,%2,%3};"
              : "+f"(acc[4 * h]), "+f"(acc[4 * h + 1]), "+f"(acc[4 * h + 2]), "+f"(acc[4 * h + 3])
              : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
        }
      }
      return;
    }
  }
#pragma unroll
  for (int k = 0; k < 16; k++) {
    const T a0 = tile_el<TA>(A, ld, g, k), a1 = tile_el<TA>(A, ld, g + 8, k);
    T bv[4];
    if constexpr (TB == TILE_FULL && sizeof(T) == 4) {
      const float2 p = *reinterpret_cast<const float2*>(B + k * ld + 2 * t),
                   q = *reinterpret_cast<const float2*>(B + k * ld + 8 + 2 * t);
      bv[0] = p.x, bv[1] = p.y, bv[2] = q.x, bv[3] = q.y;
    } else {
#pragma unroll
      for (int h = 0; h < 4; h++) bv[h] = tile_el<TB>(B, ld, k, 8 * (h >> 1) + 2 * t + (h & 1));
    }
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int j = 0; j < 2; j++) {
        acc[4 * h + j] = fma(a0, bv[2 * h + j], acc[4 * h + j]);
        acc[4 * h + 2 + j] = fma(a1, bv[2 * h + j], acc[4 * h + 2 + j]);
      }
  }
}
template <typename T>
__device__ __forceinline__ void tile_store(T* C, int ld, const T acc[8], T alpha) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int j = 0; j < 2; j++) C[(g + 8 * i) * ld + 8 * h + 2 * t + j] = alpha * acc[4 * h + 2 * i + j];
}
template <typename T>
__device__ __forceinline__ void tile_sub(T* C, int ld, const T acc[8]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int j = 0; j < 2; j++) C[(g + 8 * i) * ld + 8 * h + 2 * t + j] -= acc[4 * h + 2 * i + j];
}
// One warp: LU of the 16 x 16 tile A in place (the first n pivots count for the
// zero check); 1 / pivot to rinv.  Lane l holds row l % 16.
template <typename T>
__device__ __forceinline__ void tile_lu(T* A, int ld, int n, int boost, int* zero_flag, T* rinv) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, r = lane & 15;
  T a[16];
#pragma unroll
  for (int c = 0; c < 16; c++) a[c] = A[r * ld + c];
  T low = T(1);
#pragma unroll
  for (int k = 0; k < 16; k++) {
    T p = __shfl_sync(full, a[k], k);
    if (boost) p = boost_pivot(p);
    else if (k < n) low = fmin(low, fabs(p));
    const T inv = T(1) / p;
    if (lane == k) rinv[k] = inv;
    const T l = r > k ? a[k] * inv : T(0);
#pragma unroll
    for (int c = k + 1; c < 16; c++) a[c] = fma(-l, __shfl_sync(full, a[c], k), a[c]);
    a[k] = r > k ? l : (r == k ? p : a[k]);
  }
  if ((double)low < 1e-7 && lane == 0) atomicOr(zero_flag, 1);
  if (lane < 16) {
#pragma unroll
    for (int c = 0; c < 16; c++) A[r * ld + c] = a[c];
  }
}
// One warp: the LU in tile A replaced by L^-1 (strict lower part) and U^-1
// (upper part).  Both come from one forward recurrence: lane c < 16 solves for
// column c of L^-1 from row 0 down, lane 16 + c for column c of U^-1 from row
// 15 up, which is the same with rows and columns reversed.
template <typename T>
__device__ __forceinline__ void tile_inverses(T* A, int ld) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, r = lane & 15;
  const bool up = lane >= 16;
  T b[16], x[16];
#pragma unroll
  for (int k = 0; k < 16; k++) b[k] = A[r * ld + (up ? 15 - k : k)];
  const int e = up ? 15 - r : r;  // the unit right-hand side
#pragma unroll
  for (int i = 0; i < 16; i++) {
    const int src = up ? 31 - i : i;  // row i, or row 15 - i, of the factor
    T v = i == e ? T(1) : T(0);
#pragma unroll
    for (int k = 0; k < i; k++) v = fma(-__shfl_sync(full, b[k], src), x[k], v);
    const T d = __shfl_sync(full, b[i], src);
    x[i] = v / (up ? d : T(1));
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 16; i++) {
    const int row = up ? 15 - i : i;
    if (up ? row <= r : row > r) A[row * ld + r] = x[i];
  }
}
// One warp, 32 columns (lane's column at P, rows ld apart): P <- L^-1 P for the
// unit lower triangle of tile A.
template <typename T>
__device__ __forceinline__ void panel_lower(const T* A, T* P, int ld) {
  T x[16];
#pragma unroll
  for (int i = 0; i < 16; i++) x[i] = P[i * ld];
#pragma unroll
  for (int k = 0; k < 15; k++)
#pragma unroll
    for (int i = k + 1; i < 16; i++) x[i] = fma(-A[i * ld + k], x[k], x[i]);
#pragma unroll
  for (int i = 1; i < 16; i++) P[i * ld] = x[i];
}
// One warp, 32 rows (lane's row at P): P <- P U^-1 for the upper triangle of
// tile A, whose reciprocal pivots are rinv.
template <typename T>
__device__ __forceinline__ void panel_upper(const T* A, const T* rinv, T* P, int ld) {
  T x[16];
#pragma unroll
  for (int c = 0; c < 16; c++) x[c] = P[c];
#pragma unroll
  for (int k = 0; k < 16; k++) {
    x[k] *= rinv[k];
#pragma unroll
    for (int c = k + 1; c < 16; c++) x[c] = fma(-x[k], A[k * ld + c], x[c]);
  }
#pragma unroll
  for (int c = 0; c < 16; c++) P[c] = x[c];
}
template <typename T>
__global__ void __launch_bounds__(kLeafThreads)
k_leaf(const T* __restrict__ M, int ldm, long long sm, T* __restrict__ Li, T* __restrict__ Ui, int ldo,
       long long stride, int n, int boost, int* __restrict__ zero_flag, int tc) {
  extern __shared__ __align__(16) unsigned char leaf_raw[];
  const int nt = (n + 15) / 16, n16 = nt * 16, ld = n16 + 4;
  T* G = reinterpret_cast<T*>(leaf_raw);
  T* X = G + n16 * ld;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nw = blockDim.x >> 5;
  const T* Mb = M + blockIdx.x * sm;
  T* Lb = Li + blockIdx.x * stride;
  T* Ub = Ui + blockIdx.x * stride;
  for (int c0 = warp; c0 < n16; c0 += 4 * nw) {  // 16 loads in flight per thread
    T v[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int c = c0 + i * nw, r = lane + 32 * j;
        v[i][j] = (r < n && c < n) ? Mb[(long long)c * ldm + r] : (r == c ? T(1) : T(0));
      }
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int c = c0 + i * nw, r = lane + 32 * j;
        if (c < n16 && r < n16) G[r * ld + c] = v[i][j];
      }
  }
  __shared__ T rinv[2][16];
  __syncthreads();
  auto tile = [&](T* Z, int i, int j) { return Z + (16 * i) * ld + 16 * j; };
  auto apart = [&](int i, int j) { return tc && (i >> 1) != (j >> 1); };
  if (warp == 0) tile_lu(tile(G, 0, 0), ld, n, boost, zero_flag, rinv[0]);
  __syncthreads();
  for (int k = 0; k < nt; k++) {
    const int m = nt - 1 - k, half = (m + 1) / 2;  // panels: two tiles per warp
    if (warp < 2 * half) {
      const int o = 16 * (k + 1) + 32 * (warp % half) + lane;
      if (o < n16) {
        if (warp < half) panel_lower(tile(G, k, k), G + 16 * k * ld + o, ld);
        else panel_upper(tile(G, k, k), rinv[k & 1], G + o * ld + 16 * k, ld);
      }
    }
    __syncthreads();
    auto trail = [&](int i, int j) {
      T acc[8] = {};
      // (a pivot tile of another 32-block is a product of the recursion)
      tile_mac(tile(G, i, k), tile(G, k, j), ld, tc && (apart(i, k) || apart(j, k)), acc);
      tile_sub(tile(G, i, j), ld, acc);
    };
    if (warp == 0) {
      if (m > 0) {
        trail(k + 1, k + 1);
        __syncwarp();
        tile_lu(tile(G, k + 1, k + 1), ld, n - 16 * (k + 1), boost, zero_flag, rinv[(k + 1) & 1]);
      }
    } else if (warp == nw - 1) {
      tile_inverses(tile(G, k, k), ld);
    } else {
      for (int q = warp; q < m * m; q += nw - 2) trail(k + 1 + q / m, k + 1 + q % m);
    }
    __syncthreads();
  }
  // inverses by doubling: blocks of s tiles, pairs (2s tiles); the second of a
  // pair may be cut off by n
  for (int s = 1, ls = 0; s < nt; s *= 2, ls++) {
    const int pairs = (nt + 2 * s - 1) >> (ls + 1), per = s * s;
    for (int phase = 0; phase < 2; phase++) {
      for (int q = warp; q < pairs * per * 2; q += nw) {
        const bool up = q & 1;
        const int e = q >> 1, pr = e >> (2 * ls), i = (e >> ls) & (s - 1), j = e & (s - 1), o = pr * 2 * s, o2 = o + s;
        const int s2 = min(s, nt - o2);  // tiles of the second block
        if (s2 <= 0) continue;
        const bool t32 = tc && s > 1;
        T acc[8] = {};
        if (!up) {  // (i, j): rows o2 + i (i < s2), columns o + j
          if (i >= s2) continue;
          if (phase == 0) {  // T = L21 L11^-1
            tile_mac<TILE_FULL, TILE_UNIT_LOWER>(tile(G, o2 + i, o + j), tile(G, o + j, o + j), ld, t32, acc);
            for (int k = j + 1; k < s; k++) tile_mac(tile(G, o2 + i, o + k), tile(G, o + k, o + j), ld, t32, acc);
            tile_store(tile(X, o2 + i, o + j), ld, acc, T(1));
          } else {  // (L^-1)21 = -L22^-1 T
            for (int k = 0; k < i; k++) tile_mac(tile(G, o2 + i, o2 + k), tile(X, o2 + k, o + j), ld, t32, acc);
            tile_mac<TILE_UNIT_LOWER>(tile(G, o2 + i, o2 + i), tile(X, o2 + i, o + j), ld, t32, acc);
            tile_store(tile(G, o2 + i, o + j), ld, acc, T(-1));
          }
        } else {  // (i, j): rows o + i, columns o2 + j (j < s2)
          if (j >= s2) continue;
          if (phase == 0) {  // T = U12 U22^-1
            for (int k = 0; k < j; k++) tile_mac(tile(G, o + i, o2 + k), tile(G, o2 + k, o2 + j), ld, t32, acc);
            tile_mac<TILE_FULL, TILE_UPPER>(tile(G, o + i, o2 + j), tile(G, o2 + j, o2 + j), ld, t32, acc);
            tile_store(tile(X, o + i, o2 + j), ld, acc, T(1));
          } else {  // (U^-1)12 = -U11^-1 T
            tile_mac<TILE_UPPER>(tile(G, o + i, o + i), tile(X, o + i, o2 + j), ld, t32, acc);
            for (int k = i + 1; k < s; k++) tile_mac(tile(G, o + i, o + k), tile(X, o + k, o2 + j), ld, t32, acc);
            tile_store(tile(G, o + i, o2 + j), ld, acc, T(-1));
          }
        }
      }
      __syncthreads();
    }
  }
  for (int c = warp; c < n; c += nw)
    for (int r = lane; r < n; r += 32) {
      const T v = G[r * ld + c];
      Lb[(long long)c * ldo + r] = r > c ? v : (r == c ? T(1) : T(0));
      Ub[(long long)c * ldo + r] = r <= c ? v : T(0);
    }
}

// Largest leaf of the recursion (SAPB_LEAF: a smaller one).
template <typename T>
inline int leaf_size() {
  const char* e = std::getenv("SAPB_LEAF");
  const int v = e ? std::atoi(e) : 0;
  return v >= 32 && v <= leaf_max<T> ? v / 32 * 32 : leaf_max<T>;
}

// Batched dense matrix-vector product with an n x n column-major block:
//   y = A x            (mode 0)
//   y = c - A x        (mode 1)
// one thread per row, x staged in shared memory in tiles.  Batch b uses
// A + b*sA, x + b*sx, c + b*sc, y + b*sy (c may alias y).
template <typename T>
__global__ void __launch_bounds__(256) k_bgemv(const T* A, int ld, long long sA, const T* x, long long sx, const T* c,
                                               long long sc, T* y, long long sy, int n, int mode) {
  __shared__ T xs[256];
  const int b = blockIdx.y;
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  const T* Ab = A + b * sA;
  const T* xb = x + b * sx;
  T acc = T(0);
  for (int k0 = 0; k0 < n; k0 += 256) {
    const int kk = k0 + threadIdx.x;
    xs[threadIdx.x] = kk < n ? xb[kk] : T(0);
    __syncthreads();
    if (r < n) {
      const int kend = min(256, n - k0);
      const T* col = Ab + (long long)k0 * ld + r;
#pragma unroll 8
      for (int k = 0; k < kend; k++) acc += col[(long long)k * ld] * xs[k];
    }
    __syncthreads();
  }
  if (r < n) y[b * sy + r] = (mode == 1) ? c[b * sc + r] - acc : acc;
}

// Batched matrix-vector product over n x n column-major blocks, for the
// block sweeps and the reduced system:
//   y = A x (mode 0),  y = c - A x (mode 1; c may alias y),
// with tri = 1 (lower: row r reads columns <= r), 2 (upper: columns >= r)
// or 0 (all).  Skipped entries are exact zeros of the factors, so the
// triangular forms read half the bytes.  A CTA of 16 warps owns tiles of
// R = 32*VEC rows; lane l holds rows r0+VEC*l .. r0+VEC*l+VEC-1, so one load
// instruction of a warp is a coalesced column segment of 32*VEC elements
// (16-byte vectors when VEC*sizeof(T) = 16; VEC > 1 needs the leading
// dimension and batch stride to be multiples of VEC and A aligned to
// VEC*sizeof(T)).  The warps split the columns (8 columns in flight per
// warp) and reduce in shared memory in a fixed order.  Tiles are paired j
// with (T-1-j) so triangular work is the same for every CTA.  Batch b uses
// A + b*sA, x + b*sx, c + b*sc, y + b*sy.
// The matrix may be stored as FP16 (MT = __half, 8 rows per 16-byte load)
// with a power-of-two scale per column (see k_blocks_to_half): the kernel
// then reads x_c * cs[b*scs + c] in place of x_c and accumulates in T.
// Chains of these launches are programmatic dependent launches: every CTA
// first lets the next launch of its stream be scheduled
// (griddepcontrol.launch_dependents), then waits for the previous launch to
// complete with its writes visible (griddepcontrol.wait) before it touches
// x, c, y or the column-split scratch; the factor blocks it streams are not
// written by any launch of the apply.
constexpr int kGemvWarps = 16;
template <typename T, int VEC>
struct VecOf;
template <>
struct VecOf<double, 2> { using type = double2; };
template <>
struct VecOf<float, 4> { using type = float4; };
template <>
struct VecOf<__half, 8> { using type = uint4; };
template <typename T>
__device__ __forceinline__ T as_acc(T v) { return v; }
__device__ __forceinline__ float as_acc(__half v) { return __half2float(v); }
template <typename T>
__device__ __forceinline__ void vec_fma(const double2& a, T xv, T* acc) {
  acc[0] += a.x * xv;
  acc[1] += a.y * xv;
}
template <typename T>
__device__ __forceinline__ void vec_fma(const float4& a, T xv, T* acc) {
  acc[0] += a.x * xv;
  acc[1] += a.y * xv;
  acc[2] += a.z * xv;
  acc[3] += a.w * xv;
}
template <typename T>
__device__ __forceinline__ void vec_fma(const uint4& a, T xv, T* acc) {  // 8 x FP16
  const __half2* h = reinterpret_cast<const __half2*>(&a);
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const float2 f = __half22float2(h[q]);
    acc[2 * q] += f.x * xv;
    acc[2 * q + 1] += f.y * xv;
  }
}

//
// Column split (gridDim.z = S > 1, for grids with few tiles): CTA s takes
// the s-th contiguous slice of each of its tiles' column ranges and writes
// its R partial sums to ws[((b*ntile + tile)*S + s)*R ..]; the CTA that
// arrives last at the tile's counter (ctr, zero between launches) adds the S
// slices in order s = 0..S-1, writes y and resets the counter.  No CTA waits
// for another.
// One work item of the GEMV: tile pair `pair` (tiles pair and T-1-pair) of
// batch element b, column slice sl of S.  A, x, c, y and cs point at batch
// element b already; b only selects the column-split scratch slots.  CG:
// x and c are read through L2 (written by other CTAs of the same launch).
template <typename T, int VEC, typename MT, bool CG = false>
__device__ __forceinline__ void tgemv_item(int pair, int b, int S, int sl, const MT* Ab, int ld, const T* xb,
                                           const T* cb, T* yb, int n, int mode, int tri, T* ws, unsigned* ctr,
                                           const T* csb, T (*part)[32 * (VEC > 1 ? VEC : 2)],
                                           unsigned& last_cta) {
  constexpr int R = 32 * (VEC > 1 ? VEC : 2);
  const int ntile = (n + R - 1) / R;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // x_c, times the column scale for a scaled FP16 matrix
  auto xs = [&](int col) -> T {
    const T xc = CG ? __ldcg(xb + col) : xb[col];
    if constexpr (std::is_same<MT, T>::value) return xc;
    else return xc * csb[col];
  };
  for (int half = 0; half < 2; half++) {
    const int tile = half == 0 ? pair : ntile - 1 - pair;
    if (half == 1 && tile <= pair) break;
    const int r0 = tile * R;
    int c0 = 0, c1 = n;
    if (tri == 1) c1 = min(n, r0 + R);
    else if (tri == 2) c0 = r0;
    if (S > 1) {
      const int chunk = (c1 - c0 + S - 1) / S;
      const int a = c0 + sl * chunk;
      c1 = min(c1, a + chunk);
      c0 = min(a, c1);
    }
    // 8 independent column loads in flight per warp, then the FMAs
    constexpr int U = 8;
    constexpr int SW = kGemvWarps;  // column stride of a warp
    if constexpr (VEC > 1) {
      using V = typename VecOf<MT, VEC>::type;
      T acc[VEC];
#pragma unroll
      for (int v = 0; v < VEC; v++) acc[v] = T(0);
      const int r = r0 + VEC * lane;
      const int valid = min(VEC, max(0, n - r));
      const MT* base = Ab + r;
      int col = c0 + w;
      if (valid == VEC) {
        for (; col + (U - 1) * SW < c1; col += U * SW) {
          V a[U];
          T xv[U];
#pragma unroll
          for (int u = 0; u < U; u++) {
            a[u] = *reinterpret_cast<const V*>(base + (long long)(col + u * SW) * ld);
            xv[u] = xs(col + u * SW);
          }
#pragma unroll
          for (int u = 0; u < U; u++) vec_fma<T>(a[u], xv[u], acc);
        }
        for (; col < c1; col += SW) vec_fma<T>(*reinterpret_cast<const V*>(base + (long long)col * ld), xs(col), acc);
      } else {
        for (; col < c1; col += SW) {
          const T xv = xs(col);
          for (int v = 0; v < valid; v++) acc[v] += as_acc(base[(long long)col * ld + v]) * xv;
        }
      }
#pragma unroll
      for (int v = 0; v < VEC; v++) part[w][VEC * lane + v] = acc[v];
    } else {
      T acc0 = T(0), acc1 = T(0);
      const int ra = r0 + lane, rb = r0 + 32 + lane;
      const bool va = ra < n, vb = rb < n;
      const MT* pa = Ab + (va ? ra : 0);
      const MT* pb = Ab + (vb ? rb : 0);
      int col = c0 + w;
      for (; col + (U - 1) * SW < c1; col += U * SW) {
        T a0[U], a1[U], xv[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const long long o = (long long)(col + u * SW) * ld;
          a0[u] = va ? as_acc(pa[o]) : T(0);
          a1[u] = vb ? as_acc(pb[o]) : T(0);
          xv[u] = xs(col + u * SW);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
          acc0 += a0[u] * xv[u];
          acc1 += a1[u] * xv[u];
        }
      }
      for (; col < c1; col += SW) {
        const T xv = xs(col);
        const long long o = (long long)col * ld;
        if (va) acc0 += as_acc(pa[o]) * xv;
        if (vb) acc1 += as_acc(pb[o]) * xv;
      }
      part[w][lane] = acc0;
      part[w][32 + lane] = acc1;
    }
    __syncthreads();
    if (S == 1) {
      for (int q = threadIdx.x; q < R; q += blockDim.x) {
        const int r = r0 + q;
        T s = T(0);
#pragma unroll
        for (int k = 0; k < kGemvWarps; k++) s += part[k][q];
        if (r < n) yb[r] = (mode == 1) ? (CG ? __ldcg(cb + r) : cb[r]) - s : s;
      }
    } else {
      const long long slot = (long long)b * ntile + tile;
      for (int q = threadIdx.x; q < R; q += blockDim.x) {
        T s = T(0);
#pragma unroll
        for (int k = 0; k < kGemvWarps; k++) s += part[k][q];
        ws[(slot * S + sl) * R + q] = s;
      }
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) last_cta = (atomicAdd(&ctr[slot], 1u) == (unsigned)(S - 1));
      __syncthreads();
      if (last_cta) {
        __threadfence();
        for (int q = threadIdx.x; q < R; q += blockDim.x) {
          const int r = r0 + q;
          T s = T(0);
          for (int k = 0; k < S; k++) s += __ldcg(ws + (slot * S + k) * R + q);
          if (r < n) yb[r] = (mode == 1) ? (CG ? __ldcg(cb + r) : cb[r]) - s : s;
        }
        if (threadIdx.x == 0) ctr[slot] = 0u;
      }
    }
    __syncthreads();
  }
}

// (three CTAs per SM for the vector forms: 16 warps each, <= 42 registers)
template <typename T, int VEC, typename MT = T>
__global__ void __launch_bounds__(kGemvWarps * 32, VEC > 1 ? 3 : 1) k_tgemv(const MT* A, int ld, long long sA, const T* x, long long sx,
                                                           const T* c, long long sc, T* y, long long sy, int n,
                                                           int mode, int tri, T* ws, unsigned* ctr,
                                                           const T* cs = nullptr, long long scs = 0) {
  constexpr int R = 32 * (VEC > 1 ? VEC : 2);
  __shared__ T part[kGemvWarps][R];
  __shared__ unsigned last_cta;
  const int b = blockIdx.y;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  tgemv_item<T, VEC, MT>((int)blockIdx.x, b, (int)gridDim.z, (int)blockIdx.z, A + b * sA, ld, x + b * sx,
                         c ? c + b * sc : nullptr, y + b * sy, n, mode, tri, ws, ctr, cs ? cs + b * scs : nullptr,
                         part, last_cta);
}

// Barrier of the `n` CTAs of one group (a counter and a generation word in
// global memory, zero before the first use).  The wait is bounded: after
// kBarrierSpins polls it raises *err and returns false.
constexpr long long kBarrierSpins = 1LL << 22;
__device__ __forceinline__ bool group_barrier(unsigned* cnt, unsigned* gen, unsigned n, int* err) {
  __syncthreads();
  int ok = 1;
  if (threadIdx.x == 0) {
    const unsigned g = *reinterpret_cast<volatile unsigned*>(gen);
    __threadfence();
    if (atomicAdd(cnt, 1u) == n - 1) {
      *cnt = 0u;
      __threadfence();
      atomicAdd(gen, 1u);
    } else {
      long long it = 0;
      while (*reinterpret_cast<volatile unsigned*>(gen) == g) {
        if (++it > kBarrierSpins || *reinterpret_cast<volatile int*>(err)) {
          atomicOr(err, 1);
          ok = 0;
          break;
        }
        __nanosleep(64);
      }
    }
    __threadfence();
  }
  return __syncthreads_and(ok) != 0;
}

// One whole block sweep (x <- A_p^-1 x for every partition) as a single
// cooperative launch: partition p is served by the G CTAs of group p, which
// run its 4 nb - 2 block-row GEMVs (the steps of solve_blocks_part) with a
// group barrier between steps, S column slices per tile pair (items =
// pairs * S per step, spread over the group).  Partitions do not wait for
// each other.  Factor blocks: L_ii^-1 at Li + (p nb + i) BB, L_{i+1,i} at
// Lo + (p (nb-1) + i) BB, likewise U; their column scales (FP16 copies) at
// cs* + (block index) bs.  bar holds 2 words per partition; err is raised by
// a barrier that timed out (the kernel then returns).  stall > 0 makes every
// group barrier wait for that many CTAs more than the group has, so that the
// bounded wait runs out (tests of the timeout path only).
template <typename T, int VEC, typename MT>
__global__ void __launch_bounds__(kGemvWarps * 32, 3) k_sweep(const MT* __restrict__ Li, const MT* __restrict__ Ui,
                                                              const MT* __restrict__ Lo, const MT* __restrict__ Uo,
                                                              const T* csL, const T* csU, const T* csLo, const T* csUo,
                                                              T* x, T* y, T* t, int nb, int bs, long long BB,
                                                              long long plen, int G, int S, T* ws, unsigned* ctr,
                                                              unsigned* bar, int* err, int stall) {
  constexpr int R = 32 * (VEC > 1 ? VEC : 2);
  __shared__ T part[kGemvWarps][R];
  __shared__ unsigned last_cta;
  const int p = blockIdx.x / G, g = blockIdx.x - p * G;
  const int ntile = (bs + R - 1) / R, pairs = (ntile + 1) / 2, items = pairs * S;
  T* xp = x + p * plen;
  T* yp = y + p * plen;
  T* tp = t + p * plen;
  const long long bd = (long long)p * nb, bo = (long long)p * (nb - 1);
  const bool scaled = !std::is_same<MT, T>::value;
  const int steps = 4 * nb - 2;
  for (int s = 0; s < steps; s++) {
    const MT* A;
    const T *xv, *cv = nullptr, *cs = nullptr;
    T* yv;
    int mode = 0, tri;
    if (s < 2 * nb - 1) {  // forward: y_i = L_ii^-1 (x_i - L_{i,i-1} y_{i-1})
      const int i = (s + 1) / 2;
      if (s & 1) {
        A = Lo + (bo + i - 1) * BB;
        cs = scaled ? csLo + (bo + i - 1) * bs : nullptr;
        xv = yp + (long long)(i - 1) * bs;
        cv = xp + (long long)i * bs;
        yv = tp;
        mode = 1;
        tri = 2;
      } else {
        A = Li + (bd + i) * BB;
        cs = scaled ? csL + (bd + i) * bs : nullptr;
        xv = i > 0 ? tp : xp;
        yv = yp + (long long)i * bs;
        tri = 1;
      }
    } else {  // backward: x_i = U_ii^-1 (y_i - U_{i,i+1} x_{i+1})
      const int s2 = s - (2 * nb - 1), k = (s2 + 1) / 2, i = nb - 1 - k;
      if (s2 & 1) {
        A = Uo + (bo + i) * BB;
        cs = scaled ? csUo + (bo + i) * bs : nullptr;
        xv = xp + (long long)(i + 1) * bs;
        cv = yp + (long long)i * bs;
        yv = tp;
        mode = 1;
        tri = 1;
      } else {
        A = Ui + (bd + i) * BB;
        cs = scaled ? csU + (bd + i) * bs : nullptr;
        xv = k > 0 ? tp : yp + (long long)i * bs;
        yv = xp + (long long)i * bs;
        tri = 2;
      }
    }
    for (int it = g; it < items; it += G)
      tgemv_item<T, VEC, MT, true>(it / S, p, S, it % S, A, bs, xv, cv, yv, bs, mode, tri, ws, ctr, cs, part,
                                   last_cta);
    if (!group_barrier(bar + 2 * p, bar + 2 * p + 1, (unsigned)(G + stall), err)) return;
  }
}

// One whole block sweep for small blocks: a cluster of C CTAs per partition,
// the vectors exchanged through distributed shared memory.
//
// With blocks of a few hundred rows a step of the sweep moves some 100 KB per
// CTA, so what bounds the schedules above is the latency of a step: the first
// loads after each barrier, the partial sums and the barrier in global memory
// (10.4 us per step at 448-row blocks, 32 partitions; 2.6 us here).  Here every CTA keeps
// its share of the next step's factor block on the way into registers while
// the current step's sums are exchanged: the loads do not depend on the chain.
// Columns go round the 16 C warps of the cluster (column c to warp c mod 16 C),
// which balances the triangles; a lane holds V rows of a 32 V-row tile, one
// 16-byte load per column and tile.  Each CTA adds its warps' partial rows and
// sends them to every CTA of the cluster; one cluster barrier later all add the
// C shares in the same order, so all hold the same vector.
//
// kc: the off-diagonal factor blocks are zero outside their kc x kc corner
// (L_{i+1,i}: rows < kc, columns >= bs - kc; U_{i,i+1}: the transpose), which
// is all that is read.  bs <= 16 C JM columns and 32 V NT rows.
template <typename T, int V, typename MT, int C, int JM, int NT>
struct SweepRegs {
  using Vec = typename VecOf<MT, V>::type;
  static constexpr int W = kGemvWarps * C;  // columns per group
  static constexpr int TR = 32 * V;
  // (j, tile) is read by some column of group j: lower triangles from the
  // tile of column W j on, upper triangles up to the tile of column W j + W-1
  static constexpr bool need(bool lower, int j, int tile) {
    return lower ? tile >= W * j / TR : tile <= (W * j + W - 1) / TR;
  }
};
template <typename T, int V, typename MT, int C, int JM, int NT>
__global__ void __launch_bounds__(kGemvWarps * 32, 1)
k_sweep_cluster(const MT* __restrict__ Li, const MT* __restrict__ Ui, const MT* __restrict__ Lo,
                const MT* __restrict__ Uo, const T* __restrict__ csL, const T* __restrict__ csU,
                const T* __restrict__ csLo, const T* __restrict__ csUo, T* x, T* y, int nb, int bs, int kc,
                long long BB, long long plen) {
  using S = SweepRegs<T, V, MT, C, JM, NT>;
  using Vec = typename S::Vec;
  constexpr int W = S::W, TR = S::TR, ROWS = TR * NT;
  constexpr bool scaled = !std::is_same<MT, T>::value;
  extern __shared__ __align__(16) unsigned char sweep_raw[];
  T* part = reinterpret_cast<T*>(sweep_raw);  // [kGemvWarps][ROWS]
  T* xch = part + kGemvWarps * ROWS;          // [2][C][ROWS]
  T* xs = xch + 2 * C * ROWS;                 // [ROWS]
  const auto cluster = cooperative_groups::this_cluster();
  const int rank = (int)cluster.block_rank(), p = blockIdx.x / C;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, c0 = rank * kGemvWarps + w;
  const long long bd = (long long)p * nb, bo = (long long)p * (nb - 1);
  T* xp = x + p * plen;
  T* yp = y + p * plen;
  Vec a[JM][NT];
  T sc[JM];
  // the warp's columns of a block: rows [r0, r1), columns [k0, k1)
  auto load = [&](auto lower, const MT* A, const T* cs, int r0, int r1, int k0, int k1) {
    const MT* q = A + c0 * bs + V * lane;
#pragma unroll
    for (int j = 0; j < JM; j++, q += W * bs) {
      const int col = W * j + c0;
      const bool in = col >= k0 && col < k1;
      if constexpr (scaled) sc[j] = in ? __ldg(cs + col) : T(0);
#pragma unroll
      for (int t = 0; t < NT; t++)
        if (S::need(decltype(lower)::value, j, t)) {
          const int r = TR * t + V * lane;
          // (the triangle's empty side of a tile row is never read)
          const bool tri = decltype(lower)::value ? TR * (t + 1) > col : TR * t <= col;
          a[j][t] = in && tri && r >= r0 && r < r1 ? __ldg(reinterpret_cast<const Vec*>(q + TR * t)) : Vec{};
        }
    }
  };
  int buf = 0;
  // xs <- (c ? c - A xs : A xs) for the block held in a; c: this thread's value
  auto apply = [&](auto lower, bool minus, T cv, auto prefetch) {
    T acc[NT][V];
#pragma unroll
    for (int t = 0; t < NT; t++)
#pragma unroll
      for (int v = 0; v < V; v++) acc[t][v] = T(0);
#pragma unroll
    for (int j = 0; j < JM; j++) {
      const int col = W * j + c0;
      T xv = col < bs ? xs[col] : T(0);
      if constexpr (scaled) xv *= sc[j];
#pragma unroll
      for (int t = 0; t < NT; t++)
        if (S::need(decltype(lower)::value, j, t)) vec_fma<T>(a[j][t], xv, acc[t]);
    }
    prefetch();
#pragma unroll
    for (int t = 0; t < NT; t++)
#pragma unroll
      for (int v = 0; v < V; v++) part[w * ROWS + TR * t + V * lane + v] = acc[t][v];
    __syncthreads();
    for (int r = tid; r < bs; r += kGemvWarps * 32) {
      T s = T(0);
#pragma unroll
      for (int k = 0; k < kGemvWarps; k++) s += part[k * ROWS + r];
#pragma unroll
      for (int q = 0; q < C; q++) cluster.map_shared_rank(xch, q)[(buf * C + rank) * ROWS + r] = s;
    }
    cluster.sync();
    for (int r = tid; r < bs; r += kGemvWarps * 32) {
      T s = T(0);
#pragma unroll
      for (int q = 0; q < C; q++) s += xch[(buf * C + q) * ROWS + r];
      xs[r] = minus ? cv - s : s;
    }
    buf ^= 1;
    __syncthreads();
  };
  const std::true_type LO{};
  const std::false_type UP{};
  static_assert(ROWS <= kGemvWarps * 32, "one row per thread");
  // another CTA's shared memory may be written only once that CTA runs: all
  // have arrived before the first exchange, the first block's loads meanwhile
  // in flight
  cluster.barrier_arrive();
  load(LO, Li + bd * BB, scaled ? csL + bd * bs : nullptr, 0, bs, 0, bs);
  if (tid < bs) xs[tid] = xp[tid];
  __syncthreads();
  cluster.barrier_wait();
  for (int i = 0; i < nb; i++) {  // y_i = L_ii^-1 (x_i - L_{i,i-1} y_{i-1})
    const bool more = i + 1 < nb;
    T cv = T(0);
    apply(LO, false, T(0), [&] {
      if (more) {
        load(UP, Lo + (bo + i) * BB, scaled ? csLo + (bo + i) * bs : nullptr, 0, kc, bs - kc, bs);
        if (tid < bs) cv = xp[(long long)(i + 1) * bs + tid];
      } else {
        load(UP, Ui + (bd + i) * BB, scaled ? csU + (bd + i) * bs : nullptr, 0, bs, 0, bs);
      }
    });
    if (!more) break;
    if (rank == 0 && tid < bs) yp[(long long)i * bs + tid] = xs[tid];
    apply(UP, true, cv, [&] {
      load(LO, Li + (bd + i + 1) * BB, scaled ? csL + (bd + i + 1) * bs : nullptr, 0, bs, 0, bs);
    });
  }
  // x_i = U_ii^-1 (y_i - U_{i,i+1} x_{i+1}); rank 0 wrote the y_i: its writes
  // reach the other CTAs through the cluster barriers that followed
  for (int i = nb - 1; i >= 0; i--) {
    const bool more = i > 0;
    T cv = T(0);
    apply(UP, false, T(0), [&] {
      if (more) {
        load(LO, Uo + (bo + i - 1) * BB, scaled ? csUo + (bo + i - 1) * bs : nullptr, bs - kc, bs, 0, kc);
        if (tid < bs) cv = __ldcg(yp + (long long)(i - 1) * bs + tid);
      }
    });
    if (rank == 0 && tid < bs) xp[(long long)i * bs + tid] = xs[tid];
    if (!more) break;
    apply(LO, true, cv, [&] {
      load(UP, Ui + (bd + i - 1) * BB, scaled ? csU + (bd + i - 1) * bs : nullptr, 0, bs, 0, bs);
    });
  }
  cluster.sync();  // no CTA leaves while another may still write to it
}

// D <- L, L <- 0, U <- 0 for the bs x bs blocks of every batch element (L and D
// may have different batch strides; all 16-byte aligned)
template <typename T>
__global__ void k_take_block(T* __restrict__ L, T* __restrict__ U, long long sl, T* __restrict__ D, long long sd,
                             long long count) {
  uint4* l = reinterpret_cast<uint4*>(L + blockIdx.y * sl);
  uint4* u = reinterpret_cast<uint4*>(U + blockIdx.y * sl);
  uint4* d = reinterpret_cast<uint4*>(D + blockIdx.y * sd);
  const long long m = count * (long long)sizeof(T) / 16;
  const uint4 z = make_uint4(0, 0, 0, 0);
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < m; e += (long long)gridDim.x * blockDim.x) {
    d[e] = l[e];
    l[e] = z;
    u[e] = z;
  }
}

// rows per tile of k_tgemv<T, VEC>
template <typename T, int VEC>
constexpr int tgemv_rows() { return 32 * (VEC > 1 ? VEC : 2); }

// FP16 copies of n x n column-major blocks (block b at A + b*BB) for the
// apply, as block floating point: column c is stored as A[:, c] * 2^k_c with
// its largest magnitude in [2^14, 2^15) and cs[b*n + c] = 2^-k_c (a zero
// column gets scale 1).  Only the rows k_tgemv reads for the block's
// triangle are written: tri 1 (lower) rows from the start of the R-row tile
// holding row c, tri 2 (upper) rows up to the end of that tile.  One warp
// per column.
template <typename T, int R>
__global__ void k_blocks_to_half(const T* __restrict__ A, __half* __restrict__ H, T* __restrict__ cs, int n,
                                 long long BB, int tri) {
  const int c = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (c >= n) return;
  const long long o = (long long)blockIdx.y * BB + (long long)c * n;
  const int t0 = (c / R) * R;
  const int r0 = tri == 1 ? t0 : 0, r1 = tri == 2 ? min(n, t0 + R) : n;
  float m = 0.f;
  for (int r = r0 + lane; r < r1; r += 32) m = fmaxf(m, fabsf((float)A[o + r]));
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
  int e = 0;
  if (m > 0.f) {
    frexpf(m, &e);  // m = f * 2^e, f in [0.5, 1)
    e = max(e, -100);
  }
  const float up = m > 0.f ? ldexpf(1.f, 15 - e) : 1.f;
  for (int r = r0 + lane; r < r1; r += 32) H[o + r] = __float2half_rn((float)A[o + r] * up);
  if (lane == 0) cs[(long long)blockIdx.y * n + c] = m > 0.f ? (T)ldexpf(1.f, e - 15) : T(1);
}

// Nonzero columns of the coupling blocks: flag[blk][c] = any row of column c
// of row-major K x K block blk (blk = 2t + which) is nonzero.
template <typename T>
__global__ void k_nz_cols(const T* __restrict__ offd, int K, int* __restrict__ flag) {
  const int blk = blockIdx.y;
  const long long KK = (long long)K * K;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < K; c += gridDim.x * blockDim.x) {
    const T* M = offd + blk * KK + c;
    int nz = 0;
    for (int r = 0; r < K && !nz; r++) nz = M[(long long)r * K] != T(0);
    flag[(long long)blk * K + c] = nz;
  }
}

// Right-hand sides of the spike solves: column jj of interface t's slab is
// coupling-block column cols[t][j0+jj], placed at the interface rows
// pos[t][k] of the partition's block vector (X pre-zeroed).
template <typename T>
__global__ void k_spike_rhs(const T* __restrict__ offd, int which, int K, const int* __restrict__ cols, int ncol,
                            int j0, const int* __restrict__ pos, T* __restrict__ X, long long sX, long long plen) {
  const int jj = blockIdx.x, t = blockIdx.y;
  const int col = (j0 + jj < ncol) ? cols[(long long)t * ncol + j0 + jj] : -1;
  if (col < 0) return;
  const long long KK = (long long)K * K;
  const T* M = offd + (2LL * t + which) * KK + col;
  for (int k = threadIdx.x; k < K; k += blockDim.x)
    X[t * sX + jj * plen + pos[(long long)t * K + k]] = M[(long long)k * K];
}

// Spike tips out of the solved slab: element (k, col) of out[t], column-major
// with leading dimension ldo and batch stride so.
template <typename T>
__global__ void k_spike_tips(const T* __restrict__ X, long long sX, long long plen, const int* __restrict__ cols,
                             int ncol, int j0, const int* __restrict__ pos, int K, int ldo, long long so,
                             T* __restrict__ out) {
  const int jj = blockIdx.x, t = blockIdx.y;
  const int col = (j0 + jj < ncol) ? cols[(long long)t * ncol + j0 + jj] : -1;
  if (col < 0) return;
  for (int k = threadIdx.x; k < K; k += blockDim.x)
    out[t * so + (long long)col * ldo + k] = X[t * sX + jj * plen + pos[(long long)t * K + k]];
}

// Row-major coupling block (2t + which) -> column-major out[t] (leading
// dimension ldo, batch stride so), via 32x32 tiles.
template <typename T>
__global__ void k_couple_colmajor(const T* __restrict__ offd, int which, int K, int ldo, long long so,
                                  T* __restrict__ out) {
  __shared__ T tile[32][33];
  const int t = blockIdx.z;
  const long long KK = (long long)K * K;
  const T* M = offd + (2LL * t + which) * KK;
  T* O = out + t * so;
  const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int r = r0 + i, c = c0 + threadIdx.x;
    tile[i][threadIdx.x] = (r < K && c < K) ? M[(long long)r * K + c] : T(0);
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int c = c0 + i, r = r0 + threadIdx.x;
    if (r < K && c < K) O[(long long)c * ldo + r] = tile[threadIdx.x][i];
  }
}

// Band-order vector <-> padded block vectors of the partitions.
template <typename T>
__global__ void k_wb_to_blocks(const T* __restrict__ v, T* __restrict__ out, const int* __restrict__ pstart,
                               const int* __restrict__ psize, long long plen) {
  const int p = blockIdx.y;
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < plen; r += (long long)gridDim.x * blockDim.x)
    out[p * plen + r] = r < psize[p] ? v[pstart[p] + r] : T(0);
}
template <typename T>
__global__ void k_wb_from_blocks(const T* __restrict__ in, T* __restrict__ v, const int* __restrict__ pstart,
                                 const int* __restrict__ psize, long long plen) {
  const int p = blockIdx.y;
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < psize[p];
       r += (long long)gridDim.x * blockDim.x)
    v[pstart[p] + r] = in[p * plen + r];
}


// dst[idx[e]] = vals[e]  /  dst[e] = src[idx[e]]   (64-bit indices; idx < 0 gives 0)
template <typename T>
__global__ void k_scatter_idx(const long long* __restrict__ idx, const T* __restrict__ vals, long long m,
                              T* __restrict__ dst) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < m; e += (long long)gridDim.x * blockDim.x)
    dst[idx[e]] = vals[e];
}
template <typename T>
__global__ void k_gather_idx(const T* __restrict__ src, const long long* __restrict__ idx, long long m,
                             T* __restrict__ dst) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < m; e += (long long)gridDim.x * blockDim.x)
    dst[e] = idx[e] >= 0 ? src[idx[e]] : T(0);
}

// dst[idx[e]] = vals[e] for the K rows from `first` on of every interface's 2 K
// (first: 0 bottom of the partition before, K top of the one after)
template <typename T>
__global__ void k_iface_rows(const long long* __restrict__ idx, int K, long long rows, int first,
                             const T* __restrict__ vals, T* __restrict__ dst) {
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < rows; r += (long long)gridDim.x * blockDim.x) {
    const long long e = r / K * 2 * K + first + r % K;
    dst[idx[e]] = vals[e];
  }
}

// leftTrans into the band-order right-hand side: F[row] = T(v[gin[row]]) * sin[row]
template <typename T>
__global__ void k_wb_in(const double* __restrict__ v, const int* __restrict__ gin, const T* __restrict__ sin,
                        T* __restrict__ F, int n) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x)
    F[r] = gin ? (T)v[gin[r]] * sin[r] : (sin ? (T)v[r] * sin[r] : (T)v[r]);
}
// rightTrans out of the padded block vectors: z[sout[row]] = x(row) * cout[row]
template <typename T>
__global__ void k_wb_out(const T* __restrict__ xb, const int* __restrict__ rowpart, const int* __restrict__ pstart,
                         long long plen, const int* __restrict__ sout, const T* __restrict__ cout,
                         double* __restrict__ z, int n) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    const int p = rowpart[r];
    const T x = xb[p * plen + (r - pstart[p])];
    if (sout) z[sout[r]] = (double)(x * cout[r]);
    else z[r] = (double)(cout ? x * cout[r] : x);
  }
}

// dst[didx[e]] = src[sidx[e]]
template <typename T>
__global__ void k_move_idx(const T* __restrict__ src, const long long* __restrict__ sidx,
                           const long long* __restrict__ didx, long long m, T* __restrict__ dst) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < m; e += (long long)gridDim.x * blockDim.x)
    dst[didx[e]] = src[sidx[e]];
}

// S = I (K x K column-major with leading dimension ld, per batch element;
// padding rows zero)
template <typename T>
__global__ void k_identity(T* __restrict__ S, int K, int ld, long long stride) {
  const int b = blockIdx.y;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < (long long)ld * K;
       e += (long long)gridDim.x * blockDim.x)
    S[b * stride + e] = (e % ld == e / ld) ? T(1) : T(0);
}

}  // namespace sapb
