// The single-neighbourhood kriging classes of cyth/interpmthds.pyx:251-765
// (OrdinaryKriging, SimpleKriging, ExternalDriftKriging(_MD) and the two
// indicator classes): one station set, one variogram, a list of output
// points, every intermediate array materialised as the classes expose it.
//
// Their semantics differ from the step engine's fill_vg_var_arr matrices:
// - the station semivariogram matrix sums the components for i != j and is
//   0 on the diagonal, and a point's right-hand side is 0 at distance 0, so
//   a nugget is a discontinuity at h = 0 (the step engine takes the sill);
// - no min_vg_val cut, no sum check, no nearest-station fallback;
// - SimpleKriging's matrix is -gamma with a zero diagonal: __init__ fills it
//   with the total sill before krige() has summed it (still 0.0), and
//   krige() subtracts gamma off the diagonal (lines 397-399, 413, 432-442); its
//   right-hand side is total sill - gamma (total sill at distance 0).
//
// Kernels: the distances, the matrix and its Gauss-Jordan inverse in place of
// numpy.linalg.pinv (k_leg_system, one CTA, for small matrices; else k_leg_fill
// .. k_leg_dists, the elimination over the GPU in one cooperative launch,
// k_leg_gj, or step by step); every point's right-hand side (k_leg_rhs_fx in
// integers, k_leg_rhs in FP64); lambda = P r for every point
// as sliced tensor-core products (spi_slices.cu; without their scratch
// k_leg_lambda, an FP64 tiled contraction); k_leg_finish (a warp per point:
// estimate, variance, indicator).
#include <type_traits>

#include "spi_common.cuh"
#include "spi_gj.cuh"
#include "spi_slices.cuh"

namespace spi {

constexpr int LT = 512;        // threads of the system CTA
constexpr int LG_T = 64;       // lambda tile (points and matrix rows)
constexpr int LG_K = 16;       // lambda tile depth

__device__ __forceinline__ double leg_gamma(const spi_vg_t& vg, double d) {
  double t = 0.0;
  for (int c = 0; c < vg.n_comp; ++c) t = __dadd_rn(t, vg_eval_f64(vg.code[c], d, vg.range[c], vg.sill[c]));
  return t;
}

__device__ __forceinline__ double leg_cov(const spi_vg_t& vg, double covar, double d) {
  double t = covar;
  for (int c = 0; c < vg.n_comp; ++c) t = __dsub_rn(t, vg_eval_f64(vg.code[c], d, vg.range[c], vg.sill[c]));
  return t;
}

__device__ __forceinline__ double leg_total_sill(const spi_vg_t& vg) {
  double t = 0.0;
  for (int c = 0; c < vg.n_comp; ++c) t = __dadd_rn(t, vg.sill[c]);
  return t;
}

// Entry (i, j) of the kriging matrix.
__device__ __forceinline__ double leg_entry(int sk, const double* xi, const double* yi, int n,
                                            const double* si, const spi_vg_t& vg, int i, int j) {
  if (i < n && j < n) {
    if (i == j) return 0.0;
    const int lo = min(i, j), hi = max(i, j);
    const double g = leg_gamma(vg, dist_f64(xi[lo], yi[lo], xi[hi], yi[hi]));
    // SK: 0.0 - g_0 - g_1 ... == -(g_0 + g_1 + ...) exactly
    return sk ? -g : g;
  }
  if (i >= n && j >= n) return 0.0;
  const int st = (i < n) ? i : j;
  const int k = (i < n) ? (j - n) : (i - n);
  return (k == 0) ? 1.0 : si[(int64_t)(k - 1) * n + st];
}

// Distances, the kriging matrix and its inverse of one station set.
__global__ __launch_bounds__(LT) void k_leg_system(int sk, const double* __restrict__ xi,
                                                   const double* __restrict__ yi, int n,
                                                   const double* __restrict__ si, int n_drift,
                                                   spi_vg_t vg, double* __restrict__ dists,
                                                   double* __restrict__ lhs,
                                                   double* __restrict__ inv,
                                                   int32_t* __restrict__ status,
                                                   double* __restrict__ cond) {
  const int tid = threadIdx.x;
  const int a = sk ? 0 : 1 + n_drift;
  const int m = n + a;
  for (int64_t e = tid; e < (int64_t)m * m; e += LT) {
    const int i = (int)(e / m), j = (int)(e - (int64_t)i * m);
    double val = 0.0;
    if (i < n && j < n) {
      // (leg_entry with the distance kept: a second root took 40 us at m = 91)
      double d = 0.0;
      if (i != j) {
        const int lo = min(i, j), hi = max(i, j);
        d = dist_f64(xi[lo], yi[lo], xi[hi], yi[hi]);
        const double g = leg_gamma(vg, d);
        val = sk ? -g : g;
      }
      dists[(int64_t)i * n + j] = d;
    } else {
      val = leg_entry(sk, xi, yi, n, si, vg, i, j);
    }
    lhs[e] = val;
    inv[e] = val;
  }
  __syncthreads();
  extern __shared__ double lsm[];
  double* f = lsm;
  double* prow = lsm + m;
  int* piv = reinterpret_cast<int*>(lsm + 2 * m);
  const int fail = gj_invert<LT>(inv, m, f, prow, piv);
  // ||lhs||_F ||inv||_F >= cond_2: where it stays under 1 / (m eps), pinv's
  // cut-off removes no singular value and pinv is this inverse
  __shared__ double red[2][LT / 32];
  double sa = 0.0, sb = 0.0;
  if (!fail)
    for (int64_t e = tid; e < (int64_t)m * m; e += LT) {
      sa = fma(lhs[e], lhs[e], sa);
      sb = fma(inv[e], inv[e], sb);
    }
  for (int o = 16; o > 0; o >>= 1) {
    sa += __shfl_xor_sync(0xffffffffu, sa, o);
    sb += __shfl_xor_sync(0xffffffffu, sb, o);
  }
  if ((tid & 31) == 0) {
    red[0][tid >> 5] = sa;
    red[1][tid >> 5] = sb;
  }
  __syncthreads();
  if (tid == 0) {
    double ta = 0.0, tb = 0.0;
    for (int w = 0; w < LT / 32; ++w) {
      ta += red[0][w];
      tb += red[1][w];
    }
    status[0] = fail;
    if (cond) cond[0] = fail ? __longlong_as_double(0x7ff0000000000000LL) : sqrt(ta) * sqrt(tb);
  }
}

// ---- the same spread over the GPU ----
// One CTA updates an m x m matrix at a few FP64 operations per clock: 48 ms at
// m = 401, where the step-by-step launches below take 2 m launches of a few
// microseconds. The operations are those of gj_invert in its order, so the
// inverse is the same to the last bit. The pivots sit in the distance array,
// filled last, where it holds them; *status holds 0, or the failing step + 1.
constexpr int LS_MIN_M = 96;  // below, k_leg_gj takes longer than the one CTA (0.60 and 0.53 ms a call at 64, the same at 96)

__global__ void k_leg_fill(int sk, const double* __restrict__ xi, const double* __restrict__ yi,
                           int n, const double* __restrict__ si, int m, spi_vg_t vg,
                           double* __restrict__ lhs, double* __restrict__ inv,
                           int32_t* __restrict__ status) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *status = 0;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < (int64_t)m * m;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(e / m), j = (int)(e - (int64_t)i * m);
    lhs[e] = inv[e] = leg_entry(sk, xi, yi, n, si, vg, i, j);
  }
}

// Step k: the pivot (first row of maximum |A[i][k]|, i >= k), the row swap,
// the pivot row scaled.
__global__ __launch_bounds__(LT) void k_leg_pivot(double* __restrict__ A, int m, int k,
                                                  int32_t* __restrict__ piv,
                                                  int32_t* __restrict__ status) {
  if (*status) return;
  __shared__ double rv[LT / 32];
  __shared__ int ri[LT / 32];
  __shared__ double dk;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double best = -1.0;
  int bi = 0x7fffffff;
  auto take = [&](double x, int i) {
    if (x > best || (x == best && i < bi)) {
      best = x;
      bi = i;
    }
  };
  for (int i = k + tid; i < m; i += LT) {
    const double x = fabs(A[(int64_t)i * m + k]);
    take(isnan(x) ? __longlong_as_double(0x7ff0000000000000LL) : x, i);
  }
  for (int o = 16; o > 0; o >>= 1)
    take(__shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, bi, o));
  if (lane == 0) {
    rv[warp] = best;
    ri[warp] = bi;
  }
  __syncthreads();
  best = rv[0];
  bi = ri[0];
  for (int w = 1; w < LT / 32; ++w) take(rv[w], ri[w]);
  if (!(best > 0.0) || isinf(best)) {
    if (tid == 0) *status = k + 1;
    return;
  }
  const int p = bi;
  if (tid == 0) {
    piv[k] = p;
    dk = A[(int64_t)p * m + k];
  }
  __syncthreads();
  const double dd = dk;
  for (int j = tid; j < m; j += LT) {
    const double x = A[(int64_t)p * m + j];
    if (p != k) A[(int64_t)p * m + j] = A[(int64_t)k * m + j];
    A[(int64_t)k * m + j] = (j == k ? 1.0 : x) / dd;
  }
}

// Step k: column k eliminated from every other row, a warp per row.
__global__ __launch_bounds__(256) void k_leg_update(double* __restrict__ A, int m, int k,
                                                    const int32_t* __restrict__ status) {
  if (*status) return;
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (i >= m || i == k) return;
  const double* prow = A + (int64_t)k * m;
  double* row = A + (int64_t)i * m;
  const double fi = row[k];
  __syncwarp();  // (read before the lane of column k writes it)
  for (int j = lane; j < m; j += 32) {
    const double base = (j == k) ? 0.0 : row[j];
    row[j] = base - fi * prow[j];
  }
}

// The elimination in one cooperative launch: each CTA keeps its rows (r, r +
// B, ..) in shared memory for all steps, and rows are never moved: a row has a
// position, and a swap exchanges two positions. A step: every CTA publishes
// its largest |column k| at a position >= k together with that row; a barrier
// over the grid; every CTA picks the largest candidate (the first position on
// ties), scales its row and eliminates column k from its own. The same
// operations as k_leg_pivot and k_leg_update, which take a launch each per
// step and pass the matrix through L2 (both stay for matrices whose rows
// don't fit, m > ~1850). A step is bound by latency, the barrier's and L2's
// in a chain: m = 401 5.9 ms by launches, 3.0 so; 201 2.4, 1.2; 801 15.7, 10.5;
// 1501 41.8, 23.7.
//
// The barrier's wait is bounded: on expiry the CTA stores a status (the
// caller then takes its pseudo-inverse path from lhs) and leaves, and so do
// the others at their next wait.
struct LegCand {
  double val;  // |pivot|, NaN as infinity; -1: no row left
  int pos, pad;
};
struct LegGjWs {
  unsigned* arrived;  // zero at launch
  LegCand* cand;      // [2][B]
  double* rows;       // [2][B][m]
  int32_t* piv;
};
constexpr int LGJ_T = 256;
constexpr int LGJ_WAIT = 1 << 22;  // polls, a second or so

__global__ __launch_bounds__(LGJ_T) void k_leg_gj(double* __restrict__ A, int m, int rp,
                                                  LegGjWs W, int32_t* __restrict__ status) {
  extern __shared__ double lrows[];  // [rp][m], prow[m], f[rp], pos[rp]
  double* prow = lrows + (int64_t)rp * m;
  double* f = prow + m;
  int* pos = reinterpret_cast<int*>(f + rp);
  __shared__ int mine, gone;
  const int tid = threadIdx.x, lane = tid & 31;
  const int B = gridDim.x, b = blockIdx.x;
  const int nr = b < m ? (m - 1 - b) / B + 1 : 0;  // (<= rp)
  for (int q = 0; q < nr; ++q)
    for (int j = tid; j < m; j += LGJ_T)
      lrows[(int64_t)q * m + j] = A[(int64_t)(b + q * B) * m + j];
  for (int q = tid; q < nr; q += LGJ_T) pos[q] = b + q * B;
  if (tid == 0) gone = 0;
  __syncthreads();
  for (int k = 0; k < m; ++k) {
    LegCand* cand = W.cand + (k & 1) * B;
    double* rows = W.rows + (int64_t)(k & 1) * B * m;
    if (tid < 32) {
      double best = -1.0;
      int bi = 0x7fffffff, bq = 0;
      for (int q = lane; q < nr; q += 32) {
        const double v = lrows[(int64_t)q * m + k];
        f[q] = v;
        double x = fabs(v);
        if (isnan(x)) x = __longlong_as_double(0x7ff0000000000000LL);
        if (pos[q] >= k && (x > best || (x == best && pos[q] < bi))) {
          best = x;
          bi = pos[q];
          bq = q;
        }
      }
      for (int o = 16; o > 0; o >>= 1) {
        const double x = __shfl_xor_sync(0xffffffffu, best, o);
        const int i = __shfl_xor_sync(0xffffffffu, bi, o);
        const int q = __shfl_xor_sync(0xffffffffu, bq, o);
        if (x > best || (x == best && i < bi)) {
          best = x;
          bi = i;
          bq = q;
        }
      }
      if (lane == 0) {
        mine = best >= 0.0 ? bq : -1;
        cand[b] = LegCand{best, bi, 0};
      }
    }
    __syncthreads();
    if (mine >= 0)
      for (int j = tid; j < m; j += LGJ_T) rows[(int64_t)b * m + j] = lrows[(int64_t)mine * m + j];
    __syncthreads();
    if (tid == 0) {
      const unsigned want = (unsigned)(k + 1) * (unsigned)B;
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(W.arrived) : "memory");
      int left = LGJ_WAIT;
      unsigned seen;
      do {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(W.arrived) : "memory");
      } while (seen < want && --left > 0);
      if (seen < want) {
        gone = 1;
        *status = k + 1;
      }
    }
    __syncthreads();
    if (gone) return;
    // every warp finds the pivot for itself
    double best = -1.0;
    int p = 0x7fffffff, pb = 0;
    for (int c = lane; c < B; c += 32) {
      const double x = __ldcg(&cand[c].val);
      const int i = __ldcg(&cand[c].pos);
      if (x > best || (x == best && i < p)) {
        best = x;
        p = i;
        pb = c;
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double x = __shfl_xor_sync(0xffffffffu, best, o);
      const int i = __shfl_xor_sync(0xffffffffu, p, o);
      const int c = __shfl_xor_sync(0xffffffffu, pb, o);
      if (x > best || (x == best && i < p)) {
        best = x;
        p = i;
        pb = c;
      }
    }
    if (!(best > 0.0) || isinf(best)) {  // (the same in every CTA)
      if (b == 0 && tid == 0) *status = k + 1;
      return;
    }
    if (b == 0 && tid == 0) W.piv[k] = p;
    const double* src = rows + (int64_t)pb * m;
    const double dd = __ldcg(src + k);
    // the quotient from dd's reciprocal, rounded the same, within the
    // exponents where it is (div_rcp)
    const bool mid = best > 1e-280 && best < 1e280;
    const double dinv = __drcp_rn(dd);
    for (int j = tid; j < m; j += LGJ_T) {
      const double x = j == k ? 1.0 : __ldcg(src + j);
      const double ax = fabs(x);
      prow[j] = mid && ax < 1e280 && (ax > 1e-280 || ax == 0.0) ? div_rcp(x, dd, dinv) : x / dd;
    }
    __syncthreads();
    for (int q = 0; q < nr; ++q) {
      double* row = lrows + (int64_t)q * m;
      const int at = pos[q];
      const double fi = f[q];
      for (int j = tid; j < m; j += LGJ_T)
        row[j] = at == p ? prow[j] : (j == k ? 0.0 : row[j]) - fi * prow[j];
    }
    __syncthreads();
    for (int q = tid; q < nr; q += LGJ_T) pos[q] = pos[q] == p ? k : (pos[q] == k ? p : pos[q]);
    __syncthreads();
  }
  for (int q = 0; q < nr; ++q)
    for (int j = tid; j < m; j += LGJ_T)
      A[(int64_t)pos[q] * m + j] = lrows[(int64_t)q * m + j];
}

// Columns back into place: the reverse pivot swaps as one permutation, a row
// at a time through shared memory.
__global__ __launch_bounds__(256) void k_leg_unscramble(double* __restrict__ A, int m,
                                                        const int32_t* __restrict__ piv,
                                                        const int32_t* __restrict__ status) {
  if (*status) return;
  extern __shared__ double buf[];  // [m] a row, then the permutation
  int* at = reinterpret_cast<int*>(buf + m);
  for (int j = threadIdx.x; j < m; j += 256) at[j] = j;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int k = m - 1; k >= 0; --k) {
      const int p = piv[k];
      const int t = at[k];
      at[k] = at[p];
      at[p] = t;
    }
  for (int i = blockIdx.x; i < m; i += gridDim.x) {
    __syncthreads();
    for (int j = threadIdx.x; j < m; j += 256) buf[j] = A[(int64_t)i * m + j];
    __syncthreads();
    for (int j = threadIdx.x; j < m; j += 256) A[(int64_t)i * m + j] = buf[at[j]];
  }
}

// ||lhs||_F ||inv||_F, one CTA (a fixed order of summation).
__global__ __launch_bounds__(1024) void k_leg_norms(const double* __restrict__ lhs,
                                                    const double* __restrict__ inv, int m,
                                                    const int32_t* __restrict__ status,
                                                    double* __restrict__ cond) {
  __shared__ double red[2][32];
  const bool fail = *status != 0;
  double sa = 0.0, sb = 0.0;
  if (!fail)
    for (int64_t e = threadIdx.x; e < (int64_t)m * m; e += 1024) {
      sa = fma(lhs[e], lhs[e], sa);
      sb = fma(inv[e], inv[e], sb);
    }
  for (int o = 16; o > 0; o >>= 1) {
    sa += __shfl_xor_sync(0xffffffffu, sa, o);
    sb += __shfl_xor_sync(0xffffffffu, sb, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = sa;
    red[1][threadIdx.x >> 5] = sb;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    sa = sb = 0.0;
    for (int w = 0; w < 32; ++w) {
      sa += red[0][w];
      sb += red[1][w];
    }
    *cond = fail ? __longlong_as_double(0x7ff0000000000000LL) : sqrt(sa) * sqrt(sb);
  }
}

__global__ void k_leg_dists(const double* __restrict__ xi, const double* __restrict__ yi, int n,
                            double* __restrict__ dists) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < (int64_t)n * n;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(e / n), j = (int)(e - (int64_t)i * n);
    const int lo = min(i, j), hi = max(i, j);
    dists[e] = i == j ? 0.0 : dist_f64(xi[lo], yi[lo], xi[hi], yi[hi]);
  }
}

// rhss[k, :] of every point k.
// The same with the entries in fixed point (spi_fx.cuh), where the points
// and the variogram have that form on a grid that resolves the ranges, else by
// the FP64 formulas. A warp takes
// 32 points at a time (their grid coordinates by one lane each), its lanes
// the stations, whose grid coordinates lie in shared memory. The FP64 formula
// takes a coinciding pair (0 on the grid), deciding whether its distance is
// zero, and a spherical's or linear's semivariance under 1/32 of the sills:
// those formulas keep their relative precision down to distance 0, which a
// difference from the sill (some 2^-58 of it off) has only above that. A pair
// in a thousand or less.
//
// Bound by integer issue, some 230 operations an entry and one FP64
// operation (a structure's share of a nugget and a sill); the FP64 formulas
// take 45 at 64 issue slots each. 250 000 points of 400 stations (Exp): 8.2
// ms before, 1.07 now.
constexpr int LR_T = 256;
__global__ __launch_bounds__(LR_T) void k_leg_rhs_fx(
    int sk, const double* __restrict__ xi, const double* __restrict__ yi, int n,
    const double* __restrict__ xk, const double* __restrict__ yk, const double* __restrict__ skd,
    int64_t n_out, int n_drift, spi_vg_t vg, const FxScene* __restrict__ scene,
    double* __restrict__ rhss) {
  extern __shared__ longlong2 sxy[];  // [n]
  __shared__ FxVg f;
  __shared__ uint64_t tab[256];
  __shared__ double nug;
  __shared__ int64_t one;  // the entry at distance 0: the weights' sum
  const FxGrid gr = scene->g;
  const int tid = threadIdx.x, lane = tid & 31;
  const int m = n + (sk ? 0 : 1 + n_drift);
  if (tid == 0) {
    fx_init(f, vg, sk, 0.0, gr.q);
    if (!scene->ok || !fx_resolves(vg, gr)) f.ok = 0;
    double t = 0.0;
    for (int c = 0; c < vg.n_comp; ++c)
      if (vg.code[c] == SPI_VG_NUG) t += vg.sill[c];
    nug = t;
    one = 0;
    for (int c = 0; c < f.n; ++c) one += fx_weighed((int64_t)1 << FX_BITS, f.c[c].w);
  }
  if (tid < 256) tab[tid] = fx_exp2_entry(tid);
  __syncthreads();
  const double covar = leg_total_sill(vg);
  const int64_t w0 = ((int64_t)blockIdx.x * LR_T + tid) >> 5, nw = (int64_t)gridDim.x * LR_T / 32;
  if (f.ok)
    for (int j = tid; j < n; j += LR_T)
      sxy[j] = longlong2{fx_coord(xi[j], gr.ox, gr.q), fx_coord(yi[j], gr.oy, gr.q)};
  __syncthreads();
  const bool fx = f.ok != 0;
  const int code = f.n == 1 ? f.c[0].code : -1;
  // (an OK / EDK entry: nugget + sill (1 - rho); SK's covariance: sill rho)
  const double base = sk ? 0.0 : nug, sill = f.sill;
  const int64_t one_ = one;
  for (int64_t b = w0 * 32; b < n_out; b += nw * 32) {
    const int64_t kl = min(b + lane, n_out - 1);
    const double xl = xk[kl], yl = yk[kl];
    const int64_t cxl = fx ? fx_coord(xl, gr.ox, gr.q) : 0;
    const int64_t cyl = fx ? fx_coord(yl, gr.oy, gr.q) : 0;
    for (int u = 0; u < 32 && b + u < n_out; ++u) {
      const int64_t k = b + u;
      const int64_t cx = __shfl_sync(0xffffffffu, cxl, u), cy = __shfl_sync(0xffffffffu, cyl, u);
      double* out = rhss + k * m;
      auto exact = [&](int j) {
        const double d = dist_f64(xi[j], yi[j], xk[k], yk[k]);
        if (d == 0.0) return sk ? covar : 0.0;
        return sk ? leg_cov(vg, covar, d) : leg_gamma(vg, d);
      };
      auto row = [&](auto codec) {
        constexpr int CODE = decltype(codec)::value;
        for (int j = lane; j < n; j += 64) {
          const int j1 = min(j + 32, n - 1);
          const longlong2 s0 = sxy[j], s1 = sxy[j1];
          const FxDist d[2] = {fx_dist(cx, cy, s0.x, s0.y), fx_dist(cx, cy, s1.x, s1.y)};
          int64_t v[2];
          fx_entries<CODE, 2>(f, d, tab, v);
          double r[2];
          bool near[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            // (nests may round a unit past their sills, whose sum in FP64 is not
            // exact: the weights then add up to 2^-53 more or less than 1)
            const int64_t g = sk ? v[e] : one_ - v[e];
            near[e] = (CODE == SPI_VG_SPH || CODE < 0) && !sk && g < ((int64_t)1 << (FX_BITS - 5));
            r[e] = fma(fx_double((uint64_t)(g < 0 ? 0 : g)), sill, base);
          }
          if (d[0].S == 0 || near[0]) r[0] = exact(j);
          if (d[1].S == 0 || near[1]) r[1] = exact(j1);
          out[j] = r[0];
          if (j + 32 < n) out[j + 32] = r[1];
        }
      };
      if (!fx)
        for (int j = lane; j < n; j += 32) out[j] = exact(j);
      else if (code == SPI_VG_EXP)
        row(std::integral_constant<int, SPI_VG_EXP>{});
      else if (code == SPI_VG_GAU)
        row(std::integral_constant<int, SPI_VG_GAU>{});
      else if (code == SPI_VG_SPH)
        row(std::integral_constant<int, SPI_VG_SPH>{});
      else
        row(std::integral_constant<int, -1>{});
      for (int j = n + lane; j < m; j += 32)
        out[j] = j == n ? 1.0 : skd[(int64_t)(j - n - 1) * n_out + k];
    }
  }
}

__global__ void k_leg_rhs(int sk, const double* __restrict__ xi, const double* __restrict__ yi,
                          int n, const double* __restrict__ xk, const double* __restrict__ yk,
                          const double* __restrict__ skd, int64_t n_out, int n_drift,
                          spi_vg_t vg, double* __restrict__ rhss) {
  const int a = sk ? 0 : 1 + n_drift;
  const int m = n + a;
  const double covar = leg_total_sill(vg);
  const int64_t total = n_out * m;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = e / m;
    const int j = (int)(e - k * m);
    double v;
    if (j < n) {
      const double d = dist_f64(xi[j], yi[j], xk[k], yk[k]);
      if (d == 0.0)
        v = sk ? covar : 0.0;
      else
        v = sk ? leg_cov(vg, covar, d) : leg_gamma(vg, d);
    } else if (j == n) {
      v = 1.0;
    } else {
      v = skd[(int64_t)(j - n - 1) * n_out + k];
    }
    rhss[e] = v;
  }
}

// lambda_full[k, i] = sum_j rhss[k, j] inv[i, j]; entries i < n go to
// lambdas[k, i], the rest to mus[i - n, k]. Block: LG_T points x LG_T
// rows, 256 threads with 4 x 4 outputs each.
__global__ __launch_bounds__(256) void k_leg_lambda(const double* __restrict__ rhss,
                                                    const double* __restrict__ inv, int64_t n_out,
                                                    int n, int m, double* __restrict__ lambdas,
                                                    double* __restrict__ mus,
                                                    const int32_t* __restrict__ done,
                                                    const int32_t* __restrict__ err) {
  if (done && *done && !*err) return;  // (after a timed-out wait: computed here)
  __shared__ double rs[LG_K][LG_T + 1];
  __shared__ double ps[LG_K][LG_T + 1];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int64_t k0 = (int64_t)blockIdx.x * LG_T;
  const int i0 = blockIdx.y * LG_T;
  double acc[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = 0.0;
  for (int j0 = 0; j0 < m; j0 += LG_K) {
#pragma unroll
    for (int q = 0; q < (LG_T * LG_K) / 256; ++q) {
      const int e = tid + q * 256;
      const int row = e / LG_K, col = e % LG_K;
      const int64_t kk = k0 + row;
      const int ii = i0 + row, jj = j0 + col;
      rs[col][row] = (kk < n_out && jj < m) ? rhss[kk * m + jj] : 0.0;
      ps[col][row] = (ii < m && jj < m) ? inv[(int64_t)ii * m + jj] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int jj = 0; jj < LG_K; ++jj) {
      double rv[4], pv[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) rv[r] = rs[jj][ty * 4 + r];
#pragma unroll
      for (int c = 0; c < 4; ++c) pv[c] = ps[jj][tx * 4 + c];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = fma(rv[r], pv[c], acc[r][c]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int64_t k = k0 + ty * 4 + r;
    if (k >= n_out) continue;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = i0 + tx * 4 + c;
      if (i < n)
        lambdas[k * n + i] = acc[r][c];
      else if (i < m)
        mus[(int64_t)(i - n) * n_out + k] = acc[r][c];
    }
  }
}

// A warp per point: zk = lambda'z; OK: est = max(0, lambda'r + mu);
// SK: est = max(0, total sill - lambda'c); with ixi (the indicator
// classes' ikrige): ik = max(0, lambda'ixi), est = max(0, ik (1 - ik)).
__global__ void k_leg_finish(int sk, const double* __restrict__ zi,
                             const double* __restrict__ ixi, int n, int64_t n_out, int m,
                             spi_vg_t vg, const double* __restrict__ rhss,
                             const double* __restrict__ lambdas, const double* __restrict__ mus,
                             double* __restrict__ zk, double* __restrict__ est,
                             double* __restrict__ ik) {
  const int lane = threadIdx.x & 31;
  const int64_t k = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  if (k >= n_out) return;
  const double* lam = lambdas + k * n;
  const double* r = rhss + k * m;
  double tz = 0.0, tr = 0.0, ti = 0.0;
  for (int i = lane; i < n; i += 32) {
    const double l = lam[i];
    tz = fma(l, zi[i], tz);
    tr = fma(l, r[i], tr);
    if (ixi) ti = fma(l, ixi[i], ti);
  }
  for (int o = 16; o > 0; o >>= 1) {
    tz += __shfl_xor_sync(0xffffffffu, tz, o);
    tr += __shfl_xor_sync(0xffffffffu, tr, o);
    ti += __shfl_xor_sync(0xffffffffu, ti, o);
  }
  if (lane == 0) {
    zk[k] = tz;
    if (ixi) {
      const double p = fmax(0.0, ti);
      ik[k] = p;
      if (est) est[k] = fmax(0.0, p * (1.0 - p));
    } else if (est) {
      est[k] = sk ? fmax(0.0, leg_total_sill(vg) - tr) : fmax(0.0, tr + mus[k]);
    }
  }
}

}  // namespace spi

static int leg_check(int32_t kind, const double* xi, const double* yi, int32_t n,
                     const double* si, int32_t n_drift, const spi_vg_t* vg) {
  if (kind != SPI_KIND_OK && kind != SPI_KIND_SK && kind != SPI_KIND_EDK) return SPI_ERR_ARG;
  if (!xi || !yi || !vg || n < 1 || n_drift < 0) return SPI_ERR_ARG;
  if (vg->n_comp < 1 || vg->n_comp > SPI_MAX_VG_COMP) return SPI_ERR_VG;
  if (kind == SPI_KIND_EDK && (n_drift < 1 || !si)) return SPI_ERR_ARG;
  if (kind != SPI_KIND_EDK && n_drift != 0) return SPI_ERR_ARG;
  return SPI_OK;
}

namespace spi {
// Fewer CTAs make the barrier shorter and the updates longer. A whole
// spi_legacy_system call with an eighth as many CTAs as rows, and with a
// quarter: 2.40 and 2.25 ms at 301 rows, 3.24 and 3.65 at 401, 4.19 and 4.73 at
// 501, 5.84 and 5.78 at 601, 12.0 and 11.2 at 801.
static int leg_gj_ctas(int m, int sms) {
  const int b = m >= 350 && m <= 560 ? m / 8 : m / 4;
  return b < sms ? b : sms;
}

// k_leg_gj where its rows fit in shared memory (a quarter as many CTAs as
// rows at most, so that two published rows of each fit in the n^2 doubles of
// the workspace); false: not launched.
static bool leg_gj(double* A, int m, int n, double* ws, int32_t* piv, int32_t* status,
                   cudaStream_t st) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return false;
  const int B = leg_gj_ctas(m, sms);
  int rp = (m + B - 1) / B;
  const size_t smem = ((size_t)rp * m + m + rp) * sizeof(double) + rp * sizeof(int);
  // piv (m ints), the counter, the candidates, the rows
  const int64_t head = ((int64_t)m * 4 + 15) / 16 * 2 + 2;
  const int64_t need = head + 2 * (int64_t)B * 2 + 2 * (int64_t)B * m;
  if (smem > 200 * 1024 || need > (int64_t)n * n || reinterpret_cast<uintptr_t>(ws) % 16) return false;
  if (!smem_opt_in(k_leg_gj, smem)) return false;
  LegGjWs W;
  W.piv = piv;
  W.arrived = reinterpret_cast<unsigned*>(ws + head - 2);
  W.cand = reinterpret_cast<LegCand*>(ws + head);
  W.rows = ws + head + 4 * (int64_t)B;
  if (cudaMemsetAsync(W.arrived, 0, 16, st) != cudaSuccess) return false;
  void* args[] = {&A, &m, &rp, &W, &status};
  if (cudaLaunchCooperativeKernel((const void*)k_leg_gj, dim3(B), dim3(LGJ_T), args, smem, st) !=
      cudaSuccess) {
    cudaGetLastError();  // (no room for the grid at once: the steps one by one)
    return false;
  }
  return true;
}
}  // namespace spi

extern "C" int spi_legacy_system(int32_t kind, const double* xi, const double* yi, int32_t n,
                                 const double* si, int32_t n_drift, const spi_vg_t* vg,
                                 double* in_dists, double* lhs, double* lhs_inv,
                                 int32_t* status, double* cond, spi_stream_t stream) {
  int rc = leg_check(kind, xi, yi, n, si, n_drift, vg);
  if (rc) return rc;
  if (!in_dists || !lhs || !lhs_inv || !status) return SPI_ERR_ARG;
  const int sk = kind == SPI_KIND_SK;
  const int64_t m = (int64_t)n + (sk ? 0 : 1 + n_drift);
  const size_t smem = (size_t)m * (2 * sizeof(double) + sizeof(int));
  if (smem > 200 * 1024) return SPI_ERR_TOO_LARGE;
  // (few stations with many drifts: the one CTA)
  const bool piv_fits = m * (int64_t)sizeof(int32_t) <= (int64_t)n * n * (int64_t)sizeof(double);
  if (m >= spi::LS_MIN_M && piv_fits) {
    cudaStream_t st = (cudaStream_t)stream;
    const int mi = (int)m;
    int32_t* piv = reinterpret_cast<int32_t*>(in_dists);
    const int gx = (int)((m * m + 2047) / 2048);
    spi::k_leg_fill<<<gx, 256, 0, st>>>(sk, xi, yi, n, si, mi, *vg, lhs, lhs_inv, status);
    SPI_LAUNCH_CHECK();
    const bool one = spi::leg_gj(lhs_inv, mi, n, in_dists, piv, status, st);
    for (int k = 0; k < mi && !one; ++k) {
      spi::k_leg_pivot<<<1, spi::LT, 0, st>>>(lhs_inv, mi, k, piv, status);
      spi::k_leg_update<<<(mi + 7) / 8, 256, 0, st>>>(lhs_inv, mi, k, status);
    }
    SPI_LAUNCH_CHECK();
    const size_t us = (size_t)m * (sizeof(double) + sizeof(int));
    if (!spi::smem_opt_in(spi::k_leg_unscramble, us)) return SPI_ERR_CUDA;
    spi::k_leg_unscramble<<<mi < 304 ? mi : 304, 256, us, st>>>(lhs_inv, mi, piv, status);
    if (cond) spi::k_leg_norms<<<1, 1024, 0, st>>>(lhs, lhs_inv, mi, status, cond);
    spi::k_leg_dists<<<gx, 256, 0, st>>>(xi, yi, n, in_dists);
    SPI_LAUNCH_CHECK();
    return SPI_OK;
  }
  if (!spi::smem_opt_in(spi::k_leg_system, smem)) return SPI_ERR_CUDA;
  spi::k_leg_system<<<1, spi::LT, smem, (cudaStream_t)stream>>>(sk, xi, yi, n, si, n_drift, *vg,
                                                                in_dists, lhs, lhs_inv, status,
                                                                cond);
  SPI_LAUNCH_CHECK();
  return SPI_OK;
}

// scratch (with err_flag): lambda = P r as sliced tensor-core products.
static int leg_points(int32_t kind, const double* xi, const double* yi, const double* zi,
                      const double* ixi, int32_t n, const double* xk, const double* yk,
                      const double* sk_drift, int64_t n_out, int32_t n_drift, const spi_vg_t* vg,
                      const double* lhs_inv, double* rhss, double* lambdas, double* mus,
                      double* zk, double* est, double* ik, void* scratch, int64_t scratch_bytes,
                      int32_t* err_flag, spi_stream_t stream) {
  int rc = leg_check(kind, xi, yi, n, sk_drift, n_drift, vg);
  if (rc) return rc;
  if (n_out < 0) return SPI_ERR_ARG;
  if (n_out == 0) return SPI_OK;
  const int sk = kind == SPI_KIND_SK;
  const int a = sk ? 0 : 1 + n_drift;
  if (!zi || !xk || !yk || !lhs_inv || !rhss || !lambdas || !zk) return SPI_ERR_ARG;
  if (a > 0 && !mus) return SPI_ERR_ARG;
  if (ixi && !ik) return SPI_ERR_ARG;
  const int m = n + a;
  if ((n_out + spi::LG_T - 1) / spi::LG_T > 0x7fffffff || (n_out * 32 + 255) / 256 > 0x7fffffff)
    return SPI_ERR_TOO_LARGE;
  cudaStream_t st = (cudaStream_t)stream;
  // with the slices' scratch also the entries leave FP64 (the same sizes make
  // both pay); the stations' grid coordinates have to fit in shared memory
  const size_t sxy = (size_t)n * sizeof(longlong2);
  if (scratch && scratch_bytes >= 1024 && sxy <= 160 * 1024) {
    spi_domain_t dom = {};
    dom.n_stns = n;
    dom.stn_x = xi;
    dom.stn_y = yi;
    dom.n_cells = n_out;
    dom.cell_x = xk;
    dom.cell_y = yk;
    const spi::FxScene* scene = nullptr;
    if ((rc = spi::launch_fx_scene(dom, scratch, &scene, st))) return rc;
    if (!spi::smem_opt_in(spi::k_leg_rhs_fx, sxy)) return SPI_ERR_CUDA;
    const int64_t blocks = (n_out + spi::LR_T - 1) / spi::LR_T;
    spi::k_leg_rhs_fx<<<(unsigned)(blocks < 152 * 8 ? blocks : 152 * 8), spi::LR_T, sxy, st>>>(
        sk, xi, yi, n, xk, yk, sk_drift, n_out, n_drift, *vg, scene, rhss);
  } else {
    spi::k_leg_rhs<<<152 * 16, 256, 0, st>>>(sk, xi, yi, n, xk, yk, sk_drift, n_out, n_drift,
                                            *vg, rhss);
  }
  SPI_LAUNCH_CHECK();
  dim3 grid((unsigned)((n_out + spi::LG_T - 1) / spi::LG_T),
            (unsigned)((m + spi::LG_T - 1) / spi::LG_T));
  const int32_t* done = nullptr;
  if (scratch) {
    rc = spi::launch_slices_rows(spi::SlRows{rhss, lhs_inv, m, n, n_out, lambdas, mus}, scratch,
                                 scratch_bytes, err_flag, &done, st);
    if (rc) return rc;
  }
  spi::k_leg_lambda<<<grid, 256, 0, st>>>(rhss, lhs_inv, n_out, n, m, lambdas, mus, done,
                                          err_flag);
  SPI_LAUNCH_CHECK();
  spi::k_leg_finish<<<(unsigned)((n_out * 32 + 255) / 256), 256, 0, st>>>(
      sk, zi, ixi, n, n_out, m, *vg, rhss, lambdas, mus, zk, est, ik);
  SPI_LAUNCH_CHECK();
  return SPI_OK;
}

extern "C" int spi_legacy_points(int32_t kind, const double* xi, const double* yi,
                                 const double* zi, const double* ixi, int32_t n,
                                 const double* xk, const double* yk, const double* sk_drift,
                                 int64_t n_out, int32_t n_drift, const spi_vg_t* vg,
                                 const double* lhs_inv, double* rhss, double* lambdas,
                                 double* mus, double* zk, double* est, double* ik,
                                 spi_stream_t stream) {
  return leg_points(kind, xi, yi, zi, ixi, n, xk, yk, sk_drift, n_out, n_drift, vg, lhs_inv, rhss,
                    lambdas, mus, zk, est, ik, nullptr, 0, nullptr, stream);
}

extern "C" int spi_legacy_points_sliced(int32_t kind, const double* xi, const double* yi,
                                        const double* zi, const double* ixi, int32_t n,
                                        const double* xk, const double* yk,
                                        const double* sk_drift, int64_t n_out, int32_t n_drift,
                                        const spi_vg_t* vg, const double* lhs_inv, double* rhss,
                                        double* lambdas, double* mus, double* zk, double* est,
                                        double* ik, void* scratch, int64_t scratch_bytes,
                                        int32_t* err_flag, spi_stream_t stream) {
  if (!scratch || !err_flag) return SPI_ERR_ARG;
  return leg_points(kind, xi, yi, zi, ixi, n, xk, yk, sk_drift, n_out, n_drift, vg, lhs_inv, rhss,
                    lambdas, mus, zk, est, ik, scratch, scratch_bytes, err_flag, stream);
}

extern "C" int64_t spi_slices_one_scratch_bytes(int32_t n, int32_t rows) {
  if (n < 1 || rows < 1) return 0;
  return spi::slices_scratch_one(n, rows);
}
