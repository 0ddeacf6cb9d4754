// Cholesky factor and inverse factor of every system of a batch, spread over
// the whole GPU.
//
// Bound: FP64 issue (GB300 does about 2 FP64 FMAs per SM and clock, so
// n^3 / 3 of them on one SM are 34 ms at n = 750 where 152 SMs take 0.3 ms),
// and for the few systems of a short job the serial chain along the
// diagonal. One CTA per system, the earlier form, left all but n_sys SMs
// idle: 8 systems of 750 stations took 27 ms for the factor and 35 ms for
// its inverse (now 2.4 and 1.9 ms), 8 FP32 systems of 2900 stations 188 ms
// for the factor (now 5.1 ms, and 3.3 ms for the inverse), one of 150
// stations 0.64 and 0.48 ms (now 0.24 and 0.14 ms).
//
// Factor: right-looking, panels of 32 columns, two launches per panel over
// (tiles, systems): the panel solve, and the trailing update whose first
// tile also factors the next diagonal block, so that block's chain of square
// roots runs beside the other tiles. FP64 tiles are 32 x 32 (a tile is 16k
// cycles of one SM's FP64 pipe already), FP32 tiles 64 x 64.
// Inverse: blocks of 32 inverted by themselves, then pairs of neighbouring
// blocks of 32, 64, 128, ... joined, two products per pair,
//   [X11 0; X21 X22], X21 = -X22 (L21 X11),
// every pair, tile and system of a level in one launch: log2(n / 32) levels
// instead of n / 32 dependent block rows. L21 X11 is kept transposed in the
// mirrored (upper) block, so the inverse may overwrite its factor.
#include <cooperative_groups.h>

#include <utility>

#include "spi_factor.cuh"

namespace cg = cooperative_groups;

namespace spi {

namespace {

template <typename T>
struct Tile {
  static constexpr int TS = sizeof(T) == 8 ? 32 : 64;  // tile side
  static constexpr int MT = TS / 16;                   // outputs per thread and side
};

// The 32 x 32 (nb x nb) diagonal block in D factored by the CTA's FT
// threads; returns 0 or the 1-based failing column (the same in every
// thread). Thread (r, c8) owns row r's columns c8, c8 + 8, ...: a column's
// update is spread over all warps, since one warp alone would issue 496
// dependent FP64 instructions.
template <typename T>
__device__ int factor_diag(T (*D)[NB + 1], int nb) {
  __shared__ T rinv[NB];
  const int tid = threadIdx.x;
  const int r = tid >> 3, c8 = tid & 7;
  for (int j = 0; j < nb; ++j) {
    const T djj = D[j][j];
    if (!(djj > T(0))) return j + 1;  // not positive, or NaN
    __syncthreads();
    if (tid == 0) {
      const T l = sqrt(djj);
      D[j][j] = l;
      rinv[j] = T(1) / l;
    }
    __syncthreads();
    if (tid > j && tid < nb) D[tid][j] *= rinv[j];
    __syncthreads();
    if (r > j && r < nb) {
      const T lrj = D[r][j];
#pragma unroll
      for (int q = 0; q < NB / 8; ++q) {
        const int c = c8 + 8 * q;
        if (c > j && c <= r) D[r][c] -= lrj * D[c][j];
      }
    }
    __syncthreads();
  }
  return 0;
}

// First diagonal block of every system.
template <typename T>
__global__ __launch_bounds__(FT) void k_chol_first(spi_systems_t sys, T* __restrict__ arena,
                                                  int32_t* __restrict__ status, Gate g) {
  const int s = blockIdx.x;
  if (g.skips(s)) return;
  const SysView v = sys_view(sys, s);
  T* A = arena + v.moff;
  __shared__ T D[NB][NB + 1];
  const int nb = min(NB, v.n);
  for (int e = threadIdx.x; e < NB * NB; e += FT) {
    const int r = e / NB, c = e % NB;
    D[r][c] = (r < nb && c <= r) ? A[(int64_t)r * v.n + c] : T(0);
  }
  __syncthreads();
  const int fail = factor_diag(D, nb);
  if (threadIdx.x == 0) status[s] = fail;
  if (fail) return;
  for (int e = threadIdx.x; e < nb * nb; e += FT) {
    const int r = e / nb, c = e % nb;
    if (c <= r) A[(int64_t)r * v.n + c] = D[r][c];
  }
}

constexpr int PT = 128;          // threads of the panel solve
constexpr int PROWS = PT / 8;    // its rows: 8 lanes per row

// A21 <- A21 L11^-T below the factored diagonal block at k0: 8 lanes per
// row, each with 4 of the 32 columns; the solved entry is broadcast within
// the row's lanes and updates their later columns.
template <typename T>
__global__ __launch_bounds__(PT) void k_chol_panel(spi_systems_t sys, T* __restrict__ arena,
                                                  const int32_t* __restrict__ status, Gate g,
                                                  int k0) {
  const int s = blockIdx.y;
  if (g.skips(s) || status[s] != 0) return;
  const SysView v = sys_view(sys, s);
  const int n = v.n;
  const int rb = k0 + NB + blockIdx.x * PROWS;
  if (rb >= n) return;
  T* A = arena + v.moff;
  __shared__ T D[NB][NB + 1];
  __shared__ T rinv[NB];
  const int tid = threadIdx.x;
  for (int e = tid; e < NB * NB; e += PT) {
    const int r = e / NB, c = e % NB;
    const T x = (c <= r) ? A[(int64_t)(k0 + r) * n + k0 + c] : T(0);
    D[r][c] = x;
    if (r == c) rinv[r] = T(1) / x;
  }
  const int lane8 = tid & 7, row = rb + (tid >> 3);
  T* ar = A + (int64_t)min(row, n - 1) * n + k0;
  T x[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) x[q] = ar[lane8 + 8 * q];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < NB; ++j) {
    const T xj = __shfl_sync(0xffffffffu, x[j >> 3] * rinv[j], j & 7, 8);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = lane8 + 8 * q;
      if (q >= (j >> 3)) {
        if (c == j) x[q] = xj;
        else if (c > j) x[q] -= xj * D[c][j];
      }
    }
  }
  if (row < n)
#pragma unroll
    for (int q = 0; q < 4; ++q) ar[lane8 + 8 * q] = x[q];
}

// acc += P Q' for one K chunk of NB columns: P, Q [TS][NB + 1] in shared
// memory, thread (ty, tx) with rows ty + 16 p and columns tx + 16 q.
template <typename T>
__device__ __forceinline__ void tile_fma(const T (*P)[NB + 1], const T (*Q)[NB + 1],
                                         T (&acc)[Tile<T>::MT][Tile<T>::MT]) {
  constexpr int MT = Tile<T>::MT;
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
#pragma unroll 8
  for (int c = 0; c < NB; ++c) {
    T a[MT], b[MT];
#pragma unroll
    for (int q = 0; q < MT; ++q) {
      a[q] = P[ty + 16 * q][c];
      b[q] = Q[tx + 16 * q][c];
    }
#pragma unroll
    for (int p = 0; p < MT; ++p)
#pragma unroll
      for (int q = 0; q < MT; ++q) acc[p][q] += a[p] * b[q];
  }
}

// Row and column of tile t of a lower triangle of tiles (row-wise).
__device__ __forceinline__ void tri_tile(int t, int& ti, int& tj) {
  int i = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);
  while ((i + 1) * (i + 2) / 2 <= t) ++i;
  while (i * (i + 1) / 2 > t) --i;
  ti = i;
  tj = t - i * (i + 1) / 2;
}

// A22 -= L21 L21' on the lower triangle of the trailing matrix after the
// panel at k0; tile (0, 0)'s CTA then factors the next diagonal block.
template <typename T>
__global__ __launch_bounds__(FT) void k_chol_update(spi_systems_t sys, T* __restrict__ arena,
                                                   int32_t* __restrict__ status, Gate g,
                                                   int k0) {
  constexpr int TS = Tile<T>::TS, MT = Tile<T>::MT;
  const int s = blockIdx.y;
  if (g.skips(s) || status[s] != 0) return;
  const SysView v = sys_view(sys, s);
  const int n = v.n, r0 = k0 + NB;
  const int m = n - r0;
  if (m <= 0) return;
  const int nt = (m + TS - 1) / TS;
  if ((int)blockIdx.x >= nt * (nt + 1) / 2) return;
  int ti, tj;
  tri_tile(blockIdx.x, ti, tj);
  T* A = arena + v.moff;
  __shared__ T P[TS][NB + 1], Q[TS][NB + 1];
  const int tid = threadIdx.x;
  for (int e = tid; e < TS * NB; e += FT) {
    const int r = e / NB, c = e % NB;
    const int gi = r0 + ti * TS + r, gj = r0 + tj * TS + r;
    P[r][c] = gi < n ? A[(int64_t)gi * n + k0 + c] : T(0);
    Q[r][c] = gj < n ? A[(int64_t)gj * n + k0 + c] : T(0);
  }
  __syncthreads();
  T acc[MT][MT] = {};
  tile_fma<T>(P, Q, acc);
  const int ty = tid >> 4, tx = tid & 15;
  const bool first = blockIdx.x == 0;
  // the next diagonal block, taken over in shared memory (P is free once
  // every thread is past its products)
  __syncthreads();
#pragma unroll
  for (int p = 0; p < MT; ++p) {
    const int gi = r0 + ti * TS + ty + 16 * p;
#pragma unroll
    for (int q = 0; q < MT; ++q) {
      const int gj = r0 + tj * TS + tx + 16 * q;
      if (gi >= n || gj > gi) continue;
      const T x = A[(int64_t)gi * n + gj] - acc[p][q];
      if (first && gi < r0 + NB) P[gi - r0][gj - r0] = x;
      else A[(int64_t)gi * n + gj] = x;
    }
  }
  if (!first) return;
  __syncthreads();
  const int nb = min(NB, m);
  const int fail = factor_diag(P, nb);
  if (tid == 0 && fail) status[s] = r0 + fail;
  if (fail) return;
  for (int e = tid; e < nb * nb; e += FT) {
    const int r = e / nb, c = e % nb;
    if (c <= r) A[(int64_t)(r0 + r) * n + r0 + c] = P[r][c];
  }
}

// ---- inverse ----

// A deterministic Rademacher sign for entry i of probe k of system s.
__device__ __forceinline__ uint32_t probe_neg(int s, int k, int i) {
  uint32_t h = (uint32_t)i * 0x9E3779B1u ^ ((uint32_t)k * 0x85EBCA77u + (uint32_t)s * 0xC2B2AE3Du);
  h ^= h >> 16;
  h *= 0x7FEB352Du;
  h ^= h >> 15;
  h *= 0x846CA68Bu;
  h ^= h >> 16;
  return (h & 1u) ^ 1u;
}

constexpr int KP = 8;  // Hutchinson probes

// This CTA's share (rows i = w0, w0 + nw, ... by warps) of ||X||_F^2, or of
// sum_k |X g_k|^2 over the probes; X lower triangular. Summed over the
// warp's rows; every lane returns the warp's sum.
template <typename T>
__device__ double cond_rows(const T* X, int n, int s, int probes, int w0, int nw) {
  const int lane = threadIdx.x & 31;
  double tot = 0.0;
  for (int i = w0; i < n; i += nw) {
    const T* row = X + (int64_t)i * n;
    if (!probes) {
      T t = T(0);
      for (int j = lane; j <= i; j += 32) t += row[j] * row[j];
      double d = (double)t;
      for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
      tot += d;
      continue;
    }
    T t[KP];
#pragma unroll
    for (int k = 0; k < KP; ++k) t[k] = T(0);
    for (int j = lane; j <= i; j += 32) {
      const T x = row[j];
#pragma unroll
      for (int k = 0; k < KP; ++k) t[k] += probe_neg(s, k, j) ? -x : x;
    }
#pragma unroll
    for (int k = 0; k < KP; ++k) {
      for (int o = 16; o > 0; o >>= 1) t[k] += __shfl_xor_sync(0xffffffffu, t[k], o);
      tot += (double)t[k] * (double)t[k];
    }
  }
  return tot;
}

__device__ __forceinline__ double cond_of(int n, double x00, double f, int probes) {
  return (double)n / (x00 * x00) * (probes ? f / KP : f);
}

// Inverse of every 32 x 32 diagonal block, a lane per column of the block.
// With one block per system (max_n <= 32) the condition estimate follows
// here.
template <typename T>
__global__ __launch_bounds__(FT) void k_trinv_diag(spi_systems_t sys, const T* l_arena,
                                                  T* x_arena, const int32_t* __restrict__ status,
                                                  double* __restrict__ cond, int probes,
                                                  int single, Gate g) {
  const int s = blockIdx.y;
  if (g.skips(s)) return;
  const SysView v = sys_view(sys, s);
  const int n = v.n, i0 = blockIdx.x * NB;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (status[s] != 0) {
    if (tid == 0 && blockIdx.x == 0) cond[s] = __longlong_as_double(0x7ff0000000000000LL);
    return;
  }
  if (i0 >= n) return;
  const int nb = min(NB, n - i0);
  const T* L = l_arena + v.moff;
  T* X = x_arena + v.moff;
  __shared__ T Ld[NB][NB + 1];
  __shared__ T Xd[NB][NB + 1];
  __shared__ T rinv[NB];
  __shared__ double red[FT / 32];
  for (int e = tid; e < NB * NB; e += FT) {
    const int r = e / NB, c = e % NB;
    Ld[r][c] = (r < nb && c <= r) ? L[(int64_t)(i0 + r) * n + i0 + c] : T(0);
    Xd[r][c] = T(0);
  }
  __syncthreads();
  if (tid < nb) rinv[tid] = T(1) / Ld[tid][tid];
  __syncthreads();
  // right-looking over rows: row i of X is final once rows < i have been
  // subtracted; thread (r, c8) updates row r's columns c8 + 8 q
  const int r = tid >> 3, c8 = tid & 7;
  for (int i = 0; i < nb; ++i) {
    if (tid <= i) Xd[i][tid] = (tid == i ? T(1) : Xd[i][tid]) * rinv[i];
    __syncthreads();
    if (r > i && r < nb) {
      const T l = Ld[r][i];
#pragma unroll
      for (int q = 0; q < NB / 8; ++q) {
        const int c = c8 + 8 * q;
        if (c <= i) Xd[r][c] -= l * Xd[i][c];
      }
    }
    __syncthreads();
  }
  for (int e = tid; e < nb * nb; e += FT) {
    const int rr = e / nb, c = e % nb;
    if (c <= rr || !probes) X[(int64_t)(i0 + rr) * n + i0 + c] = (c <= rr) ? Xd[rr][c] : T(0);
  }
  if (!single) return;
  __syncthreads();
  const double t = cond_rows<T>(X, n, s, probes, warp, FT / 32);
  if (lane == 0) red[warp] = t;
  __syncthreads();
  if (tid == 0) {
    double f = 0.0;
    for (int w = 0; w < FT / 32; ++w) f += red[w];
    cond[s] = cond_of(n, (double)Xd[0][0], f, probes);
  }
}

// One product of a level: blocks of b rows at o = 2 b p (X11) and o + b
// (X22). step 0: T = L21 X11, stored transposed in the upper block; step 1:
// X21 = -X22 T. A tile of the (second block) x (first block) rectangle per
// CTA; the triangular factors' zero parts are skipped.
template <typename T>
__global__ __launch_bounds__(FT) void k_trinv_level(spi_systems_t sys, const T* l_arena,
                                                   T* x_arena,
                                                   const int32_t* __restrict__ status, int b,
                                                   int step, Gate g) {
  constexpr int TS = Tile<T>::TS, MT = Tile<T>::MT;
  const int s = blockIdx.y;
  if (g.skips(s) || status[s] != 0) return;
  const SysView v = sys_view(sys, s);
  const int n = v.n;
  const int side = (b + TS - 1) / TS;
  const int p = blockIdx.x / (side * side), t = blockIdx.x % (side * side);
  const int o = 2 * b * p, i0 = (t / side) * TS, j0 = (t % side) * TS;
  const int rows = min(b, n - o - b);  // of the second block
  if (rows <= 0 || i0 >= rows) return;
  const T* L = l_arena + v.moff;
  T* X = x_arena + v.moff;
  __shared__ T P[TS][NB + 1], Q[TS][NB + 1];
  const int tid = threadIdx.x;
  T acc[MT][MT] = {};
  // step 0 sums over k >= j (X11 lower), step 1 over k <= i (X22 lower)
  const int kb = step == 0 ? (j0 / NB) * NB : 0;
  const int ke = step == 0 ? b : min(rows, i0 + TS);
  for (int k0 = kb; k0 < ke; k0 += NB) {
    __syncthreads();
    for (int e = tid; e < TS * NB; e += FT) {
      const int r = e / NB, c = e % NB, k = k0 + c;
      // P: rows i of the left factor, Q: columns j of the right one
      T a = T(0), q = T(0);
      if (step == 0) {
        if (i0 + r < rows && k < b) a = L[(int64_t)(o + b + i0 + r) * n + o + k];
      } else {
        if (i0 + r < rows && k <= i0 + r) a = X[(int64_t)(o + b + i0 + r) * n + o + b + k];
        if (j0 + r < b && k < rows) q = X[(int64_t)(o + j0 + r) * n + o + b + k];
      }
      P[r][c] = a;
      if (step == 1) Q[r][c] = q;
    }
    if (step == 0)
      for (int e = tid; e < TS * NB; e += FT) {
        // X11's rows k along memory, transposed into Q
        const int c = e / TS, r = e % TS, k = k0 + c;
        Q[r][c] = (k < b && j0 + r <= k) ? X[(int64_t)(o + k) * n + o + j0 + r] : T(0);
      }
    __syncthreads();
    tile_fma<T>(P, Q, acc);
  }
  const int ty = tid >> 4, tx = tid & 15;
  if (step == 0) {
    // transposed store, through shared memory so that it runs along rows
    for (int h = 0; h < TS; h += NB) {  // 32 rows i at a time (P: [TS][33])
      __syncthreads();
#pragma unroll
      for (int pp = 0; pp < MT; ++pp) {
        const int i = ty + 16 * pp;
        if (i >= h && i < h + NB)
#pragma unroll
          for (int qq = 0; qq < MT; ++qq) P[tx + 16 * qq][i - h] = acc[pp][qq];
      }
      __syncthreads();
      for (int e = tid; e < TS * NB; e += FT) {
        const int j = e / NB, i = h + e % NB;
        if (i0 + i < rows && j0 + j < b)
          X[(int64_t)(o + j0 + j) * n + o + b + i0 + i] = P[j][e % NB];
      }
    }
    return;
  }
#pragma unroll
  for (int pp = 0; pp < MT; ++pp) {
    const int i = i0 + ty + 16 * pp;
#pragma unroll
    for (int qq = 0; qq < MT; ++qq) {
      const int j = j0 + tx + 16 * qq;
      if (i < rows && j < b) X[(int64_t)(o + b + i) * n + o + j] = -acc[pp][qq];
    }
  }
}

constexpr int CC = 8;     // CTAs (a cluster) per system of the condition pass
constexpr int CTH = 512;  // their threads

// The condition estimate, and (probes == 0) the strictly upper part of X
// zeroed. A cluster per system, summed in a fixed order.
template <typename T>
__global__ __cluster_dims__(CC, 1, 1) __launch_bounds__(CTH) void k_trinv_cond(
    spi_systems_t sys, T* x_arena, const int32_t* __restrict__ status,
    double* __restrict__ cond, int probes, Gate g) {
  const int s = blockIdx.y;
  if (g.skips(s) || status[s] != 0) return;  // the whole cluster alike
  const SysView v = sys_view(sys, s);
  const int n = v.n, rank = blockIdx.x;
  T* X = x_arena + v.moff;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  __shared__ double red[CTH / 32];
  __shared__ double part[CC];
  cg::cluster_group cl = cg::this_cluster();
  // (CTA 0 runs before another CTA stores into its shared memory)
  auto started = cl.barrier_arrive();
  const int nw = CC * (CTH / 32), w0 = rank * (CTH / 32) + warp;
  const double t = cond_rows<T>(X, n, s, probes, w0, nw);
  if (!probes)
    for (int i = w0; i < n; i += nw)
      for (int j = i + 1 + lane; j < n; j += 32) X[(int64_t)i * n + j] = T(0);
  if (lane == 0) red[warp] = t;
  __syncthreads();
  cl.barrier_wait(std::move(started));
  if (tid == 0) {
    double f = 0.0;
    for (int w = 0; w < CTH / 32; ++w) f += red[w];
    cl.map_shared_rank(part, 0)[rank] = f;
  }
  cl.sync();
  if (rank == 0 && tid == 0) {
    double f = 0.0;
    for (int w = 0; w < CC; ++w) f += part[w];
    cond[s] = cond_of(n, (double)X[0], f, probes);
  }
}

}  // namespace

template <typename T>
int launch_chol(const spi_systems_t& sys, T* arena, int32_t* status, Gate g, cudaStream_t st) {
  const int n = sys.max_n, S = sys.n_sys;
  k_chol_first<T><<<S, FT, 0, st>>>(sys, arena, status, g);
  SPI_LAUNCH_CHECK();
  constexpr int TS = Tile<T>::TS;
  for (int k0 = 0; k0 + NB < n; k0 += NB) {
    const int m = n - k0 - NB, nt = (m + TS - 1) / TS;
    k_chol_panel<T><<<dim3((m + PROWS - 1) / PROWS, S), PT, 0, st>>>(sys, arena, status, g, k0);
    k_chol_update<T><<<dim3(nt * (nt + 1) / 2, S), FT, 0, st>>>(sys, arena, status, g, k0);
    SPI_LAUNCH_CHECK();
  }
  return SPI_OK;
}

template <typename T>
int launch_trinv(const spi_systems_t& sys, const T* l, T* x, const int32_t* status, double* cond,
                 int probes, Gate g, cudaStream_t st) {
  const int n = sys.max_n, S = sys.n_sys;
  const int nblk = (n + NB - 1) / NB;
  k_trinv_diag<T><<<dim3(nblk, S), FT, 0, st>>>(sys, l, x, status, cond, probes, nblk == 1, g);
  SPI_LAUNCH_CHECK();
  if (nblk == 1) return SPI_OK;
  constexpr int TS = Tile<T>::TS;
  for (int b = NB; b < n; b *= 2) {
    const int pairs = (n + 2 * b - 1) / (2 * b), side = (b + TS - 1) / TS;
    for (int step = 0; step < 2; ++step)
      k_trinv_level<T><<<dim3(pairs * side * side, S), FT, 0, st>>>(sys, l, x, status, b, step, g);
    SPI_LAUNCH_CHECK();
  }
  k_trinv_cond<T><<<dim3(CC, S), CTH, 0, st>>>(sys, x, status, cond, probes, g);
  SPI_LAUNCH_CHECK();
  return SPI_OK;
}

template int launch_chol<double>(const spi_systems_t&, double*, int32_t*, Gate, cudaStream_t);
template int launch_chol<float>(const spi_systems_t&, float*, int32_t*, Gate, cudaStream_t);
template int launch_trinv<double>(const spi_systems_t&, const double*, double*, const int32_t*,
                                  double*, int, Gate, cudaStream_t);
template int launch_trinv<float>(const spi_systems_t&, const float*, float*, const int32_t*,
                                 double*, int, Gate, cudaStream_t);

}  // namespace spi
