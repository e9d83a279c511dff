// Register-window triangular sweeps of the narrow-band path (half-bandwidth
// up to kWinMaxK): the chunk solves of the apply, the chunk transfer
// matrices and carry scan, the spike tips and the reduced systems.
#pragma once

#include "precond_kernels.cuh"

namespace sapb {

// Largest half-bandwidth of the register-window kernels: the narrow path's
// own range (FP32 up to 155, FP64 up to 108; wider bands take the block path).
// The shared-memory kernels of precond_kernels.cuh take the bands that leave no
// room for packed factors, and wider ones that SAPB_WIDE_MIN_K keeps on the
// narrow path.  At these widths two K x K stages of the carry scan still fit in
// shared memory.
template <typename T>
constexpr int kWinMaxK = sizeof(T) == 8 ? 112 : 160;
// Lanes that hold a chunk's window: the warp, or half of it (two chunks per
// warp in the passes) up to K = 16, where most of 32 lanes would be past the
// band; and the register slots a lane then needs
constexpr int win_lanes(int K) { return K <= 16 ? 16 : 32; }
constexpr int win_slots(int K, int LW = 32) { return (LW - 1 + K) / LW + 1; }

// Packed factors: for every band row c its K coefficients towards the rows
// below (pkd: factor entry (c+t, c) at [c][t-1]) and towards the rows above
// (pku: (c-t, c) at [c][t-1]), each row padded with zeros to 16 bytes.  A
// sweep then streams whole aligned rows of exactly the half it needs.
template <typename T>
__host__ __device__ inline int pack_stride(int K) {
  constexpr int per = 16 / (int)sizeof(T);
  return (K + per - 1) / per * per;
}

// Coefficient staging: kStageRows packed rows per stage, kStages stages (32
// rows, some 1,000 cycles ahead of their use).  A row occupies LW R1 values of
// shared memory, zeros after its K coefficients, so that lanes left and right
// of the coefficients read zeros without a test.
constexpr int kStageRows = 8;
constexpr int kStages = 4;
constexpr int kRingRows = kStageRows * kStages;
template <typename T>
constexpr size_t win_smem(int R1, int LW = 32) { return (size_t)(32 / LW) * (kRingRows * LW * R1 + 32) * sizeof(T); }

// Forward substitution with a unit triangular band factor over the rows
// v = 0 .. m-1 in processing order, C right-hand sides per warp:
//   x(v) = rhs(v) - sum_{t=1..K} coef(v-t -> v) x(v-t),
// where coef(s -> s+t) = pk[s * pstep + t - 1] (pstep: + or - the packed row
// stride, for sweeps down or up the matrix).  With cr given, the K rows
// before the first one hold the known values cr[0..K-1] (a carry).
//
// What bounds it is the chain from row to row, so the chain is kept in
// registers: lane l holds rows base + l + 32 t (t < R1) of the window that
// the K following rows span, and four rows are resolved per step -- their
// four values are broadcast by shuffles, their 4 x 4 unit triangle is
// resolved redundantly in every lane, and each lane subtracts the four
// products from its rows.  Each row receives its updates in source order with
// one fused multiply-add each, as in a row-at-a-time solve.  The coefficients
// come through shared memory, staged by cp.async kStages - 1 stages ahead; all
// warps of the CTA share them (each has its own right-hand sides).
//
// rhs(c, v) is called once per row, by the lane that holds it, at least 32
// rows ahead of out(c, v, x), which is called once per row.  The staging area
// (win_smem) is cleared on entry.
// SOLO: the CTA is one warp.  LW < 32 (SOLO, C = 1): every LW lanes have a sweep
// of their own -- all arguments are theirs -- over windows of LW rows.
template <typename T, int R1, int C, bool SOLO, int LW = 32, typename Rhs, typename Out>
__device__ __forceinline__ void win_sweep(T* sm, const T* __restrict__ pk, long long pstep, int K, int m,
                                          const T* __restrict__ cr, Rhs rhs, Out out) {
  constexpr int RS = LW * R1, V = 16 / (int)sizeof(T), SR = kStageRows;
  static_assert(LW == 32 || (SOLO && C == 1 && LW % SR == 0), "window lanes");
  const int lane = threadIdx.x & (LW - 1), warp = SOLO ? 0 : threadIdx.x >> 5, nwarp = SOLO ? 1 : blockDim.x >> 5;
  const unsigned full = 0xffffffffu;
  const int nv = pack_stride<T>(K) / V;  // 16-byte pieces of a row, at most 64
  auto sync = [] {
    if constexpr (SOLO) __syncwarp();
    else __syncthreads();
  };
  constexpr int AREA = kRingRows * RS + 32;
  for (int e = threadIdx.x; e < AREA * (32 / LW) / V; e += blockDim.x)
    reinterpret_cast<uint4*>(sm)[e] = make_uint4(0, 0, 0, 0);
  sync();
  T* stage = sm + (LW < 32 ? (threadIdx.x & 31) / LW * AREA : 0) + 32;
  int m_all = m;  // the longest sweep of the warp
#pragma unroll
  for (int off = LW; off < 32; off *= 2) m_all = max(m_all, __shfl_xor_sync(full, m_all, off));
  const T* next = pk + lane * V;  // the lane's piece of the next row to stage
  auto issue = [&](int s0, int slot) {  // rows s0 .. s0 + SR - 1
    T* dst = stage + slot * SR * RS + lane * V;
    if (s0 + SR <= m) {
      if constexpr (SOLO) {
        if (lane < nv) {
#pragma unroll
          for (int r = 0; r < SR; r++) cp_async16(dst + r * RS, next + r * pstep);
        }
        if (LW == 32 && lane + 32 < nv) {
#pragma unroll
          for (int r = 0; r < SR; r++) cp_async16(dst + r * RS + 32 * V, next + r * pstep + 32 * V);
        }
      } else {
        for (int r = warp; r < SR; r += nwarp) {
          const T* src = next + r * pstep;
          if (lane < nv) cp_async16(dst + r * RS, src);
          if (lane + 32 < nv) cp_async16(dst + r * RS + 32 * V, src + 32 * V);
        }
      }
    } else {
      for (int r = warp; r < SR; r += nwarp)
        for (int e = lane; e < nv; e += LW) {
          T* d = dst + r * RS + (e - lane) * V;
          if (s0 + r < m) {
            cp_async16(d, next + r * pstep + (e - lane) * V);
          } else {  // rows past the end: their (unused) values stay finite
#pragma unroll
            for (int q = 0; q < V; q++) d[q] = T(0);
          }
        }
    }
    next += SR * pstep;
    cp_async_commit();
  };
#pragma unroll
  for (int q = 0; q < kStages - 1; q++) issue(q * SR, q);
  T w[C][R1];
#pragma unroll
  for (int t = 0; t < R1; t++)
#pragma unroll
    for (int c = 0; c < C; c++) {
      const int v = lane + LW * t;
      w[c][t] = v < m ? rhs(c, v) : T(0);
    }
  if (cr) {
    const T* src = pk - (long long)K * pstep + K - 1 + lane;
#pragma unroll 8
    for (int k = 0; k < K; k++) {  // carry row k is K - k rows before row 0
      const T x = cr[k];
#pragma unroll
      for (int t = 0; t + 1 < R1; t++)
        if (lane + LW * t <= k) w[0][t] = fma(-src[k * pstep - k + LW * t], x, w[0][t]);
    }
  }
  int slot = 0;
  for (int base = 0; base < m_all; base += LW) {
    T nw[C];
#pragma unroll
    for (int c = 0; c < C; c++) {
      const int v = base + LW * R1 + lane;
      nw[c] = v < m ? rhs(c, v) : T(0);
    }
    // (one stage of code: an unrolled group does not stay in the instruction
    // cache a single warp runs from)
#pragma unroll 1
    for (int h = 0; h < LW; h += SR, slot = (slot + 1) % kStages) {
      cp_async_wait<kStages - 2>();
      sync();
      issue(base + h + (kStages - 1) * SR, (slot + kStages - 1) % kStages);
#pragma unroll
      for (int b4 = 0; b4 < SR; b4 += 4) {
        const int i = h + b4;
        const T* row = stage + (slot * SR + b4) * RS;  // the four source rows
        const T* cl = row + lane - i - 1;  // lane's coefficients of row i (zeros outside 0..K-1)
        const T l10 = row[0], l20 = row[1], l30 = row[2], l21 = row[RS], l31 = row[RS + 1], l32 = row[2 * RS];
        T cf[4][R1];
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
          for (int t = 0; t < R1; t++) cf[r][t] = cl[r * RS - r + LW * t];
#pragma unroll
        for (int c = 0; c < C; c++) {
          const T x0 = __shfl_sync(full, w[c][0], i, LW);
          T x1 = __shfl_sync(full, w[c][0], i + 1, LW), x2 = __shfl_sync(full, w[c][0], i + 2, LW),
            x3 = __shfl_sync(full, w[c][0], i + 3, LW);
          x1 = fma(-l10, x0, x1);
          x2 = fma(-l21, x1, fma(-l20, x0, x2));
          x3 = fma(-l32, x2, fma(-l31, x1, fma(-l30, x0, x3)));
#pragma unroll
          for (int t = 0; t < R1; t++) {
            T a = w[c][t];
            a = fma(-cf[0][t], x0, a);
            a = fma(-cf[1][t], x1, a);
            a = fma(-cf[2][t], x2, a);
            w[c][t] = fma(-cf[3][t], x3, a);
          }
        }
      }
    }
    const int v = base + lane;
#pragma unroll
    for (int c = 0; c < C; c++) {
      if (v < m) out(c, v, w[c][0]);
#pragma unroll
      for (int t = 0; t + 1 < R1; t++) w[c][t] = w[c][t + 1];
      w[c][R1 - 1] = nw[c];
    }
  }
  cp_async_wait<0>();
  sync();
}

// Factors of partition p (band order) packed for the sweeps, and their
// pivots as a dense vector; the rows [0, rows) of every partition (all with
// rows < 0), the output starting at row p.start (or p * rows).  One warp per
// band column.
template <typename T>
__global__ void k_pack(const PartDev* __restrict__ parts, const T* __restrict__ B, int rows, int KP,
                       T* __restrict__ pkd, T* __restrict__ pku, T* __restrict__ piv) {
  const PartDev p = parts[blockIdx.y];
  const int K = p.K, lane = threadIdx.x & 31, nr = rows < 0 ? p.size : rows;
  const long long SW = 2LL * K + 1, o0 = rows < 0 ? p.start : (long long)blockIdx.y * rows;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nr; r += warps) {
    const T* c = B + p.boff + r * SW + K;
    T* d = pkd + (o0 + r) * KP;
    T* u = pku + (o0 + r) * KP;
    for (int e = lane; e < KP; e += 32) {
      d[e] = e < K ? c[e + 1] : T(0);
      u[e] = e < K ? c[-(e + 1)] : T(0);
    }
    if (lane == 0) piv[o0 + r] = c[0];
  }
}

// The three passes of a chunked partition sweep (see precond_kernels.cuh), one
// warp (up to K = 16 half a warp) per chunk.  About 50 ns per row: 1,000,000
// rows, K = 10, FP64, passes 1 / 2 / 3 65 / 140 / 66 us with a CTA per chunk and
// a barrier per row, 51 / 105 / 51 us with a warp per chunk, 39 / 66 / 35 us with
// half a warp.
// The chunk of this lane's window (past the last one: a sweep of no rows).
template <int LW>
__device__ __forceinline__ int win_chunk() {
  return (int)blockIdx.x * (32 / LW) + (LW < 32 ? (int)threadIdx.x / LW : 0);
}
template <typename T, int R1, int LW>
__global__ void __launch_bounds__(32)
k_win_pass1(const PartDev* __restrict__ parts, const ChunkDev* __restrict__ chunks, const long long* __restrict__ koff,
            const T* __restrict__ pkd, const T* __restrict__ pku, int KP, const double* __restrict__ vin, T* F,
            T* __restrict__ tails, const int* __restrict__ gin, const T* __restrict__ sin, int nch) {
  extern __shared__ __align__(16) unsigned char win_raw[];
  T* stage = reinterpret_cast<T*>(win_raw);
  const int ci = win_chunk<LW>(), c = min(ci, nch - 1);
  const ChunkDev ch = chunks[c];
  const PartDev p = parts[ch.part];
  const int K = p.K, m = ci < nch ? ch.b - ch.a : 0, dir = dir1_of(p), o = dir > 0 ? ch.a : ch.b - 1;
  T* tl = tails + koff[c];
  auto rhs = [&](int, int v) -> T {
    const int row = o + dir * v;
    if (!vin) return F[row];
    T x;
    if (gin) x = (T)vin[gin[row]] * sin[row];
    else x = sin ? (T)vin[row] * sin[row] : (T)vin[row];
    F[row] = x;
    return x;
  };
  auto out = [&](int, int v, T x) {
    if (v >= m - K) tl[v - (m - K)] = x;
  };
  win_sweep<T, R1, 1, true, LW>(stage, (dir > 0 ? pkd : pku) + (long long)o * KP, dir * KP, K, m, nullptr, rhs, out);
}

template <typename T, int R1, int LW>
__global__ void __launch_bounds__(32)
k_win_pass2(const PartDev* __restrict__ parts, const ChunkDev* __restrict__ chunks, const int* __restrict__ first1,
            const long long* __restrict__ koff, const T* __restrict__ pkd, const T* __restrict__ pku, int KP,
            const T* __restrict__ piv, const T* __restrict__ F, const T* __restrict__ carry1, T* Y,
            T* __restrict__ tails2, int nch) {
  extern __shared__ __align__(16) unsigned char win_raw[];
  T* stage = reinterpret_cast<T*>(win_raw);
  const int ci = win_chunk<LW>(), c = min(ci, nch - 1);
  const ChunkDev ch = chunks[c];
  const PartDev p = parts[ch.part];
  const int K = p.K, m = ci < nch ? ch.b - ch.a : 0, dir = dir1_of(p), o = dir > 0 ? ch.a : ch.b - 1;
  {
    auto rhs = [&](int, int v) -> T { return F[o + dir * v]; };
    auto out = [&](int, int v, T x) {
      const int row = o + dir * v;
      Y[row] = x / piv[row];
    };
    win_sweep<T, R1, 1, true, LW>(stage, (dir > 0 ? pkd : pku) + (long long)o * KP, dir * KP, K, m,
                        first1[c] ? nullptr : carry1 + koff[c], rhs, out);
  }
  const int dir2 = -dir, o2 = dir2 > 0 ? ch.a : ch.b - 1;
  T* tl = tails2 + koff[c];
  auto rhs = [&](int, int v) -> T { return Y[o2 + dir2 * v]; };
  auto out = [&](int, int v, T x) {
    if (v >= m - K) tl[v - (m - K)] = x;
  };
  win_sweep<T, R1, 1, true, LW>(stage, (dir2 > 0 ? pkd : pku) + (long long)o2 * KP, dir2 * KP, K, m, nullptr, rhs, out);
}

template <typename T, int R1, int LW>
__global__ void __launch_bounds__(32)
k_win_pass3(const PartDev* __restrict__ parts, const ChunkDev* __restrict__ chunks, const int* __restrict__ first2,
            const long long* __restrict__ koff, const T* __restrict__ pkd, const T* __restrict__ pku, int KP,
            const T* __restrict__ Y, const T* __restrict__ carry2, double* __restrict__ zout, T* __restrict__ gout,
            const int* __restrict__ sout, const T* __restrict__ cout, int nch) {
  extern __shared__ __align__(16) unsigned char win_raw[];
  T* stage = reinterpret_cast<T*>(win_raw);
  const int ci = win_chunk<LW>(), c = min(ci, nch - 1);
  const ChunkDev ch = chunks[c];
  const PartDev p = parts[ch.part];
  const int K = p.K, m = ci < nch ? ch.b - ch.a : 0, dir = -dir1_of(p), o = dir > 0 ? ch.a : ch.b - 1;
  auto rhs = [&](int, int v) -> T { return Y[o + dir * v]; };
  auto out = [&](int, int v, T x) {
    const int row = o + dir * v;
    if (zout) {
      if (sout) zout[sout[row]] = (double)(x * cout[row]);
      else zout[row] = (double)(cout ? x * cout[row] : x);
    } else {
      gout[row] = x;
    }
  };
  win_sweep<T, R1, 1, true, LW>(stage, (dir > 0 ? pkd : pku) + (long long)o * KP, dir * KP, K, m,
                      first2[c] ? nullptr : carry2 + koff[c], rhs, out);
}

// Transfer matrices in memory: T(k, u) at [k * TS + u] for carry entry k and tail
// entry u, rows padded to the scan's own thread layout (a compile-time stride up
// to K = 64) and to a multiple of four rows, zero-filled (scan_rows x TS values).
constexpr int scan_stride(int K) { return K <= 8 ? 8 : K <= 16 ? 16 : K <= 32 ? 32 : K <= 64 ? 64 : (K + 3) / 4 * 4; }
constexpr int scan_rows(int K) { return (K + 3) / 4 * 4; }
// carry entries per thread: TS * ceil(K / KG) threads take a step
constexpr int scan_kg(int K) { return K <= 8 ? 2 : K <= 16 ? 8 : K <= 32 ? 32 : K <= 64 ? 8 : K <= 128 ? 16 : 32; }
inline int scan_threads(int K) {
  return K <= 32 ? 32 : (scan_stride(K) * ((K + scan_kg(K) - 1) / scan_kg(K)) + 31) / 32 * 32;
}

// Chunk transfer matrices (see k_transfer): a CTA's warps follow C unit
// carries each through the chunk, sharing the staged coefficients; grid
// (chunk, group of carries, solve).  200,000 rows, K = 50, FP64: 5.7 -> 0.6 ms
// against one thread per carry with its window in shared memory.
template <typename T, int R1, int C>
__global__ void __launch_bounds__(512)
k_win_transfer(const PartDev* __restrict__ parts, const ChunkDev* __restrict__ chunks,
               const long long* __restrict__ toff, const T* __restrict__ pkd, const T* __restrict__ pku, int KP,
               T* __restrict__ T1, T* __restrict__ T2, int TS, const int* __restrict__ first1,
               const int* __restrict__ first2) {
  extern __shared__ __align__(16) unsigned char win_raw[];
  T* stage = reinterpret_cast<T*>(win_raw);
  const int c0 = blockIdx.x, second = blockIdx.z;
  if ((second ? first2 : first1)[c0]) return;  // no carry enters: never read
  const ChunkDev ch = chunks[c0];
  const PartDev p = parts[ch.part];
  const int K = p.K, m = ch.b - ch.a, dir = second ? -dir1_of(p) : dir1_of(p), o = dir > 0 ? ch.a : ch.b - 1;
  if ((int)blockIdx.y * C * (int)(blockDim.x >> 5) >= K) return;  // a partition narrower than the widest
  const int k0 = (blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5)) * C;
  const T* pk = (dir > 0 ? pkd : pku) + (long long)o * KP;
  const long long ps = dir * KP;
  T* Tc = (second ? T2 : T1) + toff[c0];
  auto rhs = [&](int c, int v) -> T {
    const int k = k0 + c;  // carry row k is K - k rows before the chunk
    return v <= k && k < K ? -pk[(k - K) * ps + v + K - k - 1] : T(0);
  };
  auto out = [&](int c, int v, T x) {
    if (v >= m - K && k0 + c < K) Tc[(long long)(k0 + c) * TS + v - (m - K)] = x;
  };
  // the padding of rows and columns (scan_rows x TS)
  if (blockIdx.y == 0)
    for (int e = threadIdx.x; e < scan_rows(K) * TS; e += blockDim.x)
      if (e / TS >= K || e % TS >= K) Tc[e] = T(0);
  win_sweep<T, R1, C, false>(stage, pk, ps, K, m, nullptr, rhs, out);
}

// Carry scan of one partition per CTA (see k_scan): the transfer matrices and
// tails of NB chunks at a time come into shared memory by cp.async (they are
// contiguous), one batch ahead of the chain and by warps of their own where
// there is room for them.  A chain step is a K x K product by NC threads:
// thread (g, u) holds T(g KG .., u) of the step in registers before the carry
// they multiply is known; up to K = 32 one warp takes the step (groups add by
// shuffles, no barrier but its own), above it the groups' sums meet in shared
// memory.  What bounds it is the instructions of a step, not its arithmetic:
// with runtime strides and a test per element a step took 912 cycles at K = 10,
// 1,193 at K = 64 (FP32), 1,408 at K = 50 (FP64); now 0.31 us at K = 10 and 0.54
// us at K = 64 (1.15 and 3.2 us with every load in the chain).  At K = 50 in FP64
// a batch is two chunks and its transfer sets the pace (0.83 us); a ring of six
// single-chunk stages gained 8 % there and lost 35 % in FP32.
template <typename T>
__host__ __device__ inline size_t scan_pad(size_t values) {  // to a multiple of 16 bytes
  constexpr size_t per = 16 / sizeof(T);
  return (values + per - 1) / per * per;
}
// values of one batch: NB matrices, NB tails
template <typename T>
inline size_t scan_batch(int K, int NB) {
  return (size_t)scan_rows(K) * scan_stride(K) * NB + scan_pad<T>((size_t)K * NB);
}
// maxK: the widest partition's (its strides hold for all); TSC: scan_stride(maxK)
// when it is a compile-time class, else 0
template <typename T, int KG, int TSC>
__global__ void __launch_bounds__(TSC == 32 ? 512 : 1024)
k_win_scan(const PartDev* __restrict__ parts, const int* __restrict__ pchunk0, const int* __restrict__ pnchunk,
           const long long* __restrict__ koff, const long long* __restrict__ toff, const T* __restrict__ Tm,
           const T* __restrict__ tails, T* __restrict__ carry, int which, int ts, int NC, int NB) {
  const PartDev p = parts[blockIdx.x];
  const int K = p.K, c0 = pchunk0[blockIdx.x], nc = pnchunk[blockIdx.x];
  if (nc <= 1) return;
  const int dir = (which == 1) ? dir1_of(p) : -dir1_of(p);
  extern __shared__ __align__(16) unsigned char win_raw[];
  constexpr bool WARP = TSC > 0 && TSC <= 32;
  const int TS = TSC ? TSC : ts, KR = scan_rows(K), KT = KR * TS;
  const size_t TO = (size_t)KT * NB, SB = TO + scan_pad<T>((size_t)K * NB);
  T* st = reinterpret_cast<T*>(win_raw);
  T* sig = st + 2 * SB;                            // the carry, zeros up to KZ
  const int G = (K + KG - 1) / KG, KZ = WARP ? 32 : G * KG;
  T* red = sig + KZ;                               // G * TS
  const int tid = threadIdx.x, NT = blockDim.x;
  const int u = TSC ? tid % (TSC ? TSC : 1) : tid % ts, g = TSC ? tid / (TSC ? TSC : 1) : tid / ts;
  const bool act = WARP || g < G;
  const T* Tp = Tm + toff[c0];
  const T* tp = tails + koff[c0];
  T* cp = carry + koff[c0];
  constexpr int V = 16 / (int)sizeof(T);
  for (int e = tid; e < KZ; e += NT) sig[e] = T(0);
  const int lt = NT > NC ? tid - NC : tid, LT = NT > NC ? NT - NC : NT;  // the copying threads
  // batch b: steps b NB .. ; chunks [lo, lo + cnt) of the partition
  auto batch = [&](int b, int& lo, int& cnt) {
    const int s0 = b * NB;
    cnt = min(NB, nc - 1 - s0);
    lo = dir > 0 ? s0 : nc - s0 - cnt;
  };
  auto issue = [&](int b) {
    int lo, cnt;
    batch(b, lo, cnt);
    if (cnt > 0 && lt >= 0) {
      T* d = st + (b & 1) * SB;
      const T* src = Tp + (long long)lo * KT;
      for (int e = lt * V; e < cnt * KT; e += LT * V) cp_async16(d + e, src + e);
      const T* ts_ = tp + (long long)lo * K;
      for (int e = lt; e < cnt * K; e += LT) cp_async_val<T>(d + TO + e, ts_ + e);
    }
    cp_async_commit();
  };
  auto sync = [&] {
    if constexpr (WARP) __syncwarp();
    else asm volatile("bar.sync 1, %0;" ::"r"(NC) : "memory");
  };
  issue(0);
  for (int b = 0; b * NB < nc - 1; b++) {
    cp_async_wait<0>();
    __syncthreads();
    issue(b + 1);
    if (tid >= NC) continue;
    int lo, cnt;
    batch(b, lo, cnt);
    const int dj = dir > 0 ? 1 : -1;
    int j = dir > 0 ? 0 : cnt - 1;  // chunk lo + j
    const T* tq = st + (b & 1) * SB + (long long)j * KT + g * KG * TS + u;
    const T* lq = st + (b & 1) * SB + TO + j * K + (u < K ? u : 0);
    T* cq = cp + (long long)(lo + j + dj) * K + u;
    T tv[KG], tl = T(0);
    auto load = [&] {
#pragma unroll
      for (int k = 0; k < KG; k += KG < 4 ? KG : 4)
        if (act && g * KG + k < KR) {
#pragma unroll
          for (int i = 0; i < (KG < 4 ? KG : 4); i++) tv[k + i] = tq[(k + i) * TS];
        }
      tl = *lq;
    };
#pragma unroll
    for (int k = 0; k < KG; k++) tv[k] = T(0);
    load();
    for (int q = 0; q < cnt; q++) {
      T acc[4] = {T(0), T(0), T(0), T(0)};
      if (b + q > 0) {  // (no carry enters the first chunk)
        const T* sg = sig + g * KG;
#pragma unroll
        for (int k = 0; k < KG; k += KG < 4 ? KG : 4)
          if (act && g * KG + k < KR) {
            T x[4];
            if constexpr (KG % 4 == 0 && sizeof(T) == 4) {
              const float4 f = *reinterpret_cast<const float4*>(sg + k);
              x[0] = f.x, x[1] = f.y, x[2] = f.z, x[3] = f.w;
            } else if constexpr (KG % 4 == 0) {
              const double2 f = *reinterpret_cast<const double2*>(sg + k), h = *reinterpret_cast<const double2*>(sg + k + 2);
              x[0] = f.x, x[1] = f.y, x[2] = h.x, x[3] = h.y;
            } else {
#pragma unroll
              for (int i = 0; i < KG; i++) x[i] = sg[i];
            }
#pragma unroll
            for (int i = 0; i < (KG < 4 ? KG : 4); i++) acc[i] = fma(tv[k + i], x[i], acc[i]);
          }
      }
      T v = (acc[0] + acc[1]) + (acc[2] + acc[3]);
      const T tail = tl;
      tq += (long long)dj * KT;
      lq += dj * K;
      if (q + 1 < cnt) load();
      if constexpr (WARP) {
#pragma unroll
        for (int off = TSC; off < 32; off *= 2) v += __shfl_xor_sync(0xffffffffu, v, off);
        v += tail;
        sync();  // all lanes have read the carry
      } else {
        if (act) red[g * TS + u] = v;
        sync();
        if (g == 0 && u < K) {
          T s0 = tail, s1 = T(0);
          int r = 0;
#pragma unroll 4
          for (; r + 1 < G; r += 2) {
            s0 += red[r * TS + u];
            s1 += red[(r + 1) * TS + u];
          }
          if (r < G) s0 += red[r * TS + u];
          v = s0 + s1;
        }
      }
      if (g == 0 && u < K) {
        *cq = v;
        sig[u] = v;
      }
      cq += dj * K;
      sync();
    }
  }
}

// Spike tips of the LU_UL method (see k_spikes_luul): grid (interface, tip,
// group of columns), each warp C columns through the K-row corner.  V from
// the LU corner at the bottom of partition i, W from the UL corner at the top
// of partition i+1, packed apart (k_pack with rows = K) in pkd2 / pku2 / piv2.
template <typename T, int R1, int C>
__global__ void __launch_bounds__(256)
k_win_spikes_luul(const PartDev* __restrict__ parts, const T* __restrict__ pkd, const T* __restrict__ pku,
                  const T* __restrict__ piv, const T* __restrict__ pkd2, const T* __restrict__ pku2,
                  const T* __restrict__ piv2, const T* __restrict__ offd, T* V, T* Wm, int K, int KP) {
  extern __shared__ __align__(16) unsigned char win_raw[];
  T* stage = reinterpret_cast<T*>(win_raw);
  const int i = blockIdx.x, which = blockIdx.y;
  const int k0 = (blockIdx.z * (blockDim.x >> 5) + (threadIdx.x >> 5)) * C;
  const long long KK = (long long)K * K;
  const T* d = which ? pkd2 : pkd;
  const T* u = which ? pku2 : pku;
  const T* pv = which ? piv2 : piv;
  const long long lo = which ? (long long)(i + 1) * K : parts[i + 1].start - K;  // first corner row
  const T* M = offd + (2 * i + which) * KK;
  T* X = (which ? Wm : V) + i * KK;
  const int dir = which == 0 ? 1 : -1;  // of the first solve
  auto row = [&](int v, int dr) { return dr > 0 ? v : K - 1 - v; };
  {
    auto rhs = [&](int c, int v) -> T { return k0 + c < K ? M[row(v, dir) * K + k0 + c] : T(0); };
    auto out = [&](int c, int v, T x) {
      const int r = row(v, dir);
      if (k0 + c < K) X[r * K + k0 + c] = x / pv[lo + r];
    };
    win_sweep<T, R1, C, false>(stage, (dir > 0 ? d : u) + (lo + row(0, dir)) * KP, dir * KP, K, K, nullptr, rhs, out);
  }
  auto rhs = [&](int c, int v) -> T { return k0 + c < K ? X[row(v, -dir) * K + k0 + c] : T(0); };
  auto out = [&](int c, int v, T x) {
    if (k0 + c < K) X[row(v, -dir) * K + k0 + c] = x;
  };
  win_sweep<T, R1, C, false>(stage, (dir < 0 ? d : u) + (lo + row(0, -dir)) * KP, -dir * KP, K, K, nullptr, rhs, out);
}

// Spike tips from LU factors of both neighbours (see k_spikes_luonly and
// k_spikes_var): the columns of a coupling block swept through the whole
// partition from the first interface row on, one column contiguous in
// scratch, and the interface rows read back.  iface null: the constant band
// (the bottom K rows of partition i, the top K rows of partition i+1, the
// former through the corner alone).  A 60,013-row half-bandwidth 37 FP32
// band in 16 partitions: 24.6 ms with one thread per column, 0.36 ms now.
template <typename T, int R1, int C>
__global__ void __launch_bounds__(256)
k_win_spikes_lu(const PartDev* __restrict__ parts, const T* __restrict__ pkd, const T* __restrict__ pku,
                const T* __restrict__ piv, int KP, const T* __restrict__ offd, const int* __restrict__ iface, T* __restrict__ V, T* __restrict__ Wm, T* scratch, long long stride,
                int K) {
  extern __shared__ __align__(16) unsigned char win_raw[];
  T* stage = reinterpret_cast<T*>(win_raw);
  const int i = blockIdx.x, which = blockIdx.y, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int cg0 = blockIdx.z * nw * C;  // the CTA's first column
  const int k0 = cg0 + (threadIdx.x >> 5) * C;
  const long long KK = (long long)K * K;
  const PartDev p = parts[i + which];
  const T* M = offd + (2 * i + which) * KK;
  T* out_m = (which ? Wm : V) + i * KK;
  const int* map = iface ? iface + (long long)i * 2 * K + (which ? K : 0) : nullptr;
  const int np = p.size, Kp = p.K;
  auto pos = [&](int r) { return map ? map[r] - p.start : (which ? r : np - K + r); };
  __shared__ int any, low;
  if (threadIdx.x == 0) {
    any = 0;
    low = np;
  }
  __syncthreads();
  bool nz = false;
  const int ncol = min(nw * C, K - cg0);
  for (int e = threadIdx.x; e < ncol * K; e += blockDim.x) nz |= M[(e / ncol) * K + cg0 + e % ncol] != T(0);
  int lw = np;
  for (int r = threadIdx.x; r < K; r += blockDim.x) lw = min(lw, pos(r));
  if (nz) any = 1;
  atomicMin(&low, lw);
  __syncthreads();
  if (!any) {  // zero columns have zero tips
    for (int e = threadIdx.x; e < ncol * K; e += blockDim.x) out_m[(e / ncol) * K + cg0 + e % ncol] = T(0);
    return;
  }
  const int lo = low, M_rows = np - lo;
  // x[c * stride + row]; the constant band's V needs K rows a column only
  // (spike_scratch)
  T* x = scratch + ((long long)(2 * i + which) * K + k0) * stride;
  if (!map) {
    x = scratch + ((long long)i * K + k0) * stride;
    if (!which) {
      x = scratch + (long long)gridDim.x * K * stride + ((long long)i * K + k0) * K - lo;
      stride = K;
    }
  }
  for (int c = 0; c < C && k0 + c < K; c++) {
    T* xc = x + c * stride;
    for (int j = lo + lane; j < np; j += 32) xc[j] = T(0);
    __syncwarp();
    for (int r = lane; r < K; r += 32) xc[pos(r)] = M[r * K + k0 + c];
  }
  __syncwarp();
  {
    auto rhs = [&](int c, int v) -> T { return k0 + c < K ? x[c * stride + lo + v] : T(0); };
    auto out = [&](int c, int v, T y) {
      if (k0 + c < K) x[c * stride + lo + v] = y / piv[p.start + lo + v];
    };
    win_sweep<T, R1, C, false>(stage, pkd + (long long)(p.start + lo) * KP, KP, Kp, M_rows, nullptr, rhs, out);
  }
  auto rhs = [&](int c, int v) -> T { return k0 + c < K ? x[c * stride + np - 1 - v] : T(0); };
  auto out = [&](int c, int v, T y) {
    if (k0 + c < K) x[c * stride + np - 1 - v] = y;
  };
  win_sweep<T, R1, C, false>(stage, pku + (long long)(p.start + np - 1) * KP, -KP, Kp, M_rows, nullptr, rhs, out);
  for (int c = 0; c < C && k0 + c < K; c++)
    for (int r = lane; r < K; r += 32) out_m[r * K + k0 + c] = x[c * stride + pos(r)];
}

// values of k_win_spikes_lu's scratch
inline size_t spike_scratch(int nI, int K, int maxsz, bool var_band) {
  return (size_t)nI * K * (var_band ? 2 * (size_t)maxsz : (size_t)maxsz + K);
}

// Reduced system of each interface (see k_reduced_factor) with S in shared
// memory (leading dimension odd): the product I - W V, then the elimination
// with two barriers per pivot and no global traffic in the chain.
template <typename T>
inline size_t reduced_smem(int K) { return (size_t)K * (K | 1) * sizeof(T); }
template <typename T>
__global__ void __launch_bounds__(512)
k_win_reduced_factor(const T* __restrict__ V, const T* __restrict__ Wm, T* __restrict__ S, int K, int do_boost) {
  extern __shared__ __align__(16) unsigned char win_raw[];
  T* s = reinterpret_cast<T*>(win_raw);
  const int i = blockIdx.x, tid = threadIdx.x, NT = blockDim.x, ld = K | 1;
  const int tx = tid & 31, ty = tid >> 5, ny = NT >> 5;
  const long long KK = (long long)K * K;
  const T* Vi = V + i * KK;
  const T* Wi = Wm + i * KK;
  for (int r = ty; r < K; r += ny)
    for (int c = tx; c < K; c += 32) {
      T acc = (r == c) ? T(1) : T(0);
#pragma unroll 8
      for (int k = 0; k < K; k++) acc = fma(-Wi[r * K + k], Vi[k * K + c], acc);
      s[r * ld + c] = acc;
    }
  for (int j = 0; j < K; j++) {
    __syncthreads();
    T p = s[j * ld + j];
    if (do_boost) p = boost_pivot(p);
    for (int r = j + 1 + ty; r < K; r += ny) {
      const T l = s[r * ld + j] / p;
      for (int c = j + 1 + tx; c < K; c += 32) s[r * ld + c] = fma(-l, s[j * ld + c], s[r * ld + c]);
      __syncwarp();
      if (tx == 0) s[r * ld + j] = l;
    }
  }
  __syncthreads();
  for (int r = ty; r < K; r += ny) {
    T p = s[r * ld + r];
    if (do_boost) p = boost_pivot(p);
    for (int c = tx; c < K; c += 32)
      S[i * KK + r * K + c] = c > r ? s[r * ld + c] / p : (c == r ? p : s[r * ld + c]);
  }
}

// Reduced solve and purification of each interface (see k_reduced_apply),
// with S in shared memory, the triangular solves by one warp in registers
// (rows lane + 32 t, each step's value broadcast by a shuffle) and the four
// products with V, W and the coupling blocks by all warps, one row per warp
// at a time.
template <typename T, int R>
__global__ void __launch_bounds__(512)
k_win_reduced_apply(const PartDev* __restrict__ parts, const T* __restrict__ V, const T* __restrict__ Wm,
                    const T* __restrict__ S, const T* __restrict__ offd, const T* __restrict__ Gv, T* __restrict__ F,
                    int K, const int* __restrict__ iface) {
  extern __shared__ __align__(16) unsigned char win_raw[];
  const int ld = K | 1;
  T* s = reinterpret_cast<T*>(win_raw);
  T* xb = s + K * ld;
  T* z = xb + K;
  T* x1 = z + K;
  const int i = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const long long KK = (long long)K * K;
  const int st = parts[i + 1].start;
  const T* Vi = V + i * KK;
  const T* Wi = Wm + i * KK;
  const T* Si = S + i * KK;
  const T* Bm = offd + (2 * i) * KK;
  const T* Cm = offd + (2 * i + 1) * KK;
  const int* map = iface ? iface + (long long)i * 2 * K : nullptr;
  auto pos_b = [&](int q) { return map ? map[q] : st - K + q; };
  auto pos_t = [&](int q) { return map ? map[K + q] : st + q; };
  for (int r = warp; r < K; r += nw)
    for (int c = lane; c < K; c += 32) cp_async_val<T>(s + r * ld + c, Si + r * K + c);
  cp_async_commit();
  if (tid < K) xb[tid] = Gv[pos_b(tid)];
  __syncthreads();
  // done(r, A[r] . x) for the K rows, four per warp at a time (their loads in
  // flight together)
  constexpr int RB = 4;
  auto rows_dot = [&](const T* A, const T* x, auto done) {
    for (int r0 = warp * RB; r0 < K; r0 += nw * RB) {
      T a[RB];
#pragma unroll
      for (int q = 0; q < RB; q++) a[q] = T(0);
#pragma unroll
      for (int t = 0; t < R; t++) {
        const int c = lane + 32 * t;
        const T xc = c < K ? x[c] : T(0);
#pragma unroll
        for (int q = 0; q < RB; q++)
          if (c < K && r0 + q < K) a[q] = fma(A[(r0 + q) * K + c], xc, a[q]);
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int q = 0; q < RB; q++) a[q] += __shfl_xor_sync(0xffffffffu, a[q], off);
#pragma unroll
      for (int q = 0; q < RB; q++)
        if (lane == q && r0 + q < K) done(r0 + q, a[q]);
    }
  };
  rows_dot(Wi, xb, [&](int r, T a) { z[r] = Gv[pos_t(r)] - a; });
  cp_async_wait<0>();
  __syncthreads();
  if (warp == 0) {
    T w[R];
#pragma unroll
    for (int t = 0; t < R; t++) w[t] = lane + 32 * t < K ? z[lane + 32 * t] : T(0);
#pragma unroll
    for (int tj = 0; tj < R; tj++)
#pragma unroll 4
      for (int l = 0; l < 32 && 32 * tj + l < K; l++) {
        const int j = 32 * tj + l;
        const T zj = __shfl_sync(0xffffffffu, w[tj], l);
#pragma unroll
        for (int t = tj; t < R; t++) {
          const int r = lane + 32 * t;
          if (r > j && r < K) w[t] = fma(-s[r * ld + j], zj, w[t]);
        }
      }
#pragma unroll
    for (int t = 0; t < R; t++) {
      const int r = lane + 32 * t;
      if (r < K) w[t] /= s[r * ld + r];
    }
#pragma unroll
    for (int tj = R - 1; tj >= 0; tj--)
#pragma unroll 4
      for (int l = min(31, K - 1 - 32 * tj); l >= 0; l--) {
        const int j = 32 * tj + l;
        const T zj = __shfl_sync(0xffffffffu, w[tj], l);
#pragma unroll
        for (int t = 0; t <= tj; t++) {
          const int r = lane + 32 * t;
          if (r < j) w[t] = fma(-s[r * ld + j], zj, w[t]);
        }
      }
#pragma unroll
    for (int t = 0; t < R; t++)
      if (lane + 32 * t < K) z[lane + 32 * t] = w[t];
  }
  __syncthreads();
  rows_dot(Vi, z, [&](int r, T a) { x1[r] = xb[r] - a; });
  // (a partition of fewer than 2 K rows has rows that belong to both of its
  // interfaces, whose CTAs run side by side)
  rows_dot(Bm, z, [&](int r, T b) { atomicAdd(&F[pos_b(r)], -b); });
  __syncthreads();
  rows_dot(Cm, x1, [&](int r, T a) { atomicAdd(&F[pos_t(r)], -a); });
}

}  // namespace sapb
