// FP64 build + factorisation of every kriging system of a batch, and the
// per-step dual weights.
//
// Replaces, for all systems at once, what interp/steps.py:170-243 (LHS
// assembly from the precomputed cell/station variogram matrices) and
// interp/steps.py:350-352 (numpy.linalg.pinv of the LHS) do per group:
// the LHS is built straight from station coordinates (fused distance +
// variogram, never materialising the N x N matrix of every variogram), put
// in covariance form A = s*11' - Gamma, and factored A = L L' in FP64. The
// Lagrange / drift rows are handled by a Schur complement S = F'A^-1 F.
//
// GB300's FP64 pipe is narrow (about 2 DFMA per SM per clock), so these
// kernels are FP64-issue bound, not memory bound. The factor and its inverse
// (spi_chol.cu) and the dual vectors (spi_duals.cu) spread over the GPU; the
// assembly, the drift check, the exact inverse of small systems and the host
// side are here.
#include "spi_common.cuh"
#include "spi_factor.cuh"
#include "spi_gj.cuh"
#include "spi_saddle.cuh"

namespace spi {

// The exact-inverse path's elimination over the whole GPU (spi_gj_multi.cu).
int launch_gj_multi(const spi_domain_t& dom, const spi_systems_t& sys, const spi_krige_ws_t& ws,
                    double cond_max, int pinv_on, cudaStream_t st);

// Resolves routes 3 / 4 left by k_gj (spi_pinv.cu).
int launch_pinv(const spi_domain_t& dom, const spi_systems_t& sys, const spi_krige_ws_t& ws,
                cudaStream_t st);

// Sum of one value per thread over the block (all threads call it).
__device__ double block_sum(double t, double* red) {
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[warp] = t;
  __syncthreads();
  double r = 0.0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) r += red[w];
  __syncthreads();
  return r;
}

// A[i, j] for i >= j. The reference fills the upper triangle of the full
// station matrix from dists[lo, hi] and mirrors it (cyth/interpmthds.pyx:
// 196-226); with ascending station lists the entry (i, j), i > j, is the
// mirror of (j, i), whose distance is dist(stn[j], stn[i]).
// A variogram of nuggets alone. The reference's semivariogram is then the
// total sill at every distance, h = 0 included (cyth/interpmthds.pyx:38-84),
// so its saddle matrix [[c J, F], [F', 0]] has rank 2 a and numpy's pinv
// gives its minimum-norm solution: lambda = F (F'F)^-1 f with zero
// multipliers (OK: the mean of the values; EDK: the drifts' least-squares
// fit), and for SK (a zero covariance matrix) lambda = 0.
__device__ __forceinline__ bool nug_only(const spi_vg_t& vg) {
  for (int c = 0; c < vg.n_comp; ++c)
    if (vg.code[c] != SPI_VG_NUG) return false;
  return vg.n_comp > 0;
}

// The system matrix of the Cholesky path: the covariance form sh - Gamma
// (SK: the covariances). For a nugget-only variogram the covariance form
// is the zero matrix; the identity takes its place: the dual form then
// gives lambda = c - F nu with F'lambda = f, and with the covariances c = 0
// that is the minimum-norm solution above (SK: lambda = c = 0), whatever
// the matrix's size.
// full: both triangles (the refinement's products read rows). Bound by FP64
// issue, some 45 operations an entry: a pair is evaluated once and its
// divisions by the range are products with correctly rounded reciprocals,
// the same values. 8 systems of 2900 stations, both triangles: 7.4 ms
// before, 3.3 now; 60 of 375, lower triangles: 0.60, 0.49.
__global__ __launch_bounds__(256) void k_build_sys(spi_domain_t dom, spi_systems_t sys,
                                                   double* __restrict__ l_arena,
                                                   double* __restrict__ shift_out, int full) {
  __shared__ VgPre pre;
  const int s = blockIdx.y;
  SysView v = sys_view(sys, s);
  const spi_vg_t vg = sys.vg[s];
  const int sk = sys.kind == SPI_KIND_SK;
  const double sh = sk ? 0.0 : total_sill(vg);
  const bool nug = nug_only(vg);
  if (blockIdx.x == 0 && threadIdx.x == 0) shift_out[s] = sh;
  if (threadIdx.x == 0) pre.init(vg);
  __syncthreads();
  // (outside, r^3 or its reciprocal may leave FP64's range)
  bool mid = true;
  for (int c = 0; c < vg.n_comp; ++c) mid = mid && vg.range[c] > 1e-60 && vg.range[c] < 1e60;
  double* A = l_arena + v.moff;
  const int64_t nn = (int64_t)v.n * v.n;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nn;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(e / v.n), j = (int)(e - (int64_t)i * v.n);
    if (j > i) {
      if (!full) A[e] = 0.0;  // (full: with its mirror)
      continue;
    }
    double x;
    if (nug) {
      x = (i == j) ? 1.0 : 0.0;
    } else {
      // (i, j) and its mirror from the same distance: dists[lo, hi]
      const int si = v.idx[i], sj = v.idx[j];
      const double d = dist_f64(dom.stn_x[sj], dom.stn_y[sj], dom.stn_x[si], dom.stn_y[si]);
      // (a product by a reciprocal takes an infinite distance, or one of 2^497 on
      // whose cube is, for no number)
      const double g = mid && __double2hiint(d) < 0x5f000000 ? pre.fill(d, sk, dom.min_vg_val)
                                                             : vg_fill_f64(vg, d, sk, dom.min_vg_val);
      x = sk ? g : __dsub_rn(sh, g);
    }
    A[e] = x;
    if (full && j < i) A[(int64_t)j * v.n + i] = x;
  }
}

// Exact-inverse path. Systems whose Cholesky failed, or whose condition
// estimate exceeds cond_max, get the reference's own saddle matrix
// [[Gamma, F], [F', 0]] (interp/steps.py:170-243; SK: the covariance
// matrix) inverted in place by Gauss-Jordan with partial pivoting (first
// row of maximum |pivot|), columns unscrambled in reverse pivot order.
// That is numpy.linalg.pinv (interp/steps.py:351) whenever pinv's
// singular-value cut-off (1e-15 s_max, numpy's default) removes nothing,
// which holds while ||M||_F ||P||_F <= 1e15; cond[s] receives that
// product. With
// pinv_on, systems of m <= SPI_PINV_MAX_M rows above it (or with a zero
// pivot) are left to k_pinv (route 3: inverse valid, 4: Gauss-Jordan
// failed). Dynamic shared memory: m pivot factors + m pivot indices.
__global__ __launch_bounds__(FT) void k_gj(spi_domain_t dom, spi_systems_t sys,
                                          double* __restrict__ l_arena,
                                          const int32_t* __restrict__ status,
                                          double* __restrict__ cond,
                                          int32_t* __restrict__ route, double cond_max,
                                          int pinv_on, Gate g) {
  const int s = blockIdx.x;
  const int tid = threadIdx.x;
  if (g.skips(s)) return;
  if (status[s] == 0 && cond[s] <= cond_max) {
    if (tid == 0) route[s] = 0;
    return;
  }
  SysView v = sys_view(sys, s);
  const int n = v.n;
  const int sk = sys.kind == SPI_KIND_SK;
  const int a = extra_rows(sys.kind, dom.n_drift);
  const int m = n + a;
  const spi_vg_t vg = sys.vg[s];
  double* A = l_arena + v.moff;
  extern __shared__ double gsm[];
  double* f = gsm;                                   // [m]
  double* prow = gsm + m;                            // [m] the scaled pivot row
  int* piv = reinterpret_cast<int*>(gsm + 2 * m);    // [m]
  __shared__ double red[FT / 32];
  // saddle matrix, full storage, and its squared Frobenius norm
  double fm = 0.0;
  for (int64_t e = tid; e < (int64_t)m * m; e += FT) {
    const int i = (int)(e / m), j = (int)(e - (int64_t)i * m);
    const double val = saddle_entry(dom, vg, v.idx, n, sk, i, j);
    A[e] = val;
    fm += val * val;
  }
  fm = block_sum(fm, red);
  const int fail = gj_invert<FT>(A, m, f, prow, piv);
  double fp = 0.0;
  if (!fail)
    for (int64_t e = tid; e < (int64_t)m * m; e += FT) fp += A[e] * A[e];
  fp = block_sum(fp, red);
  if (tid == 0) {
    const double cg = sqrt(fm) * sqrt(fp);
    cond[s] = fail ? __longlong_as_double(0x7ff0000000000000LL) : cg;
    // pinv (default rcond 1e-15) cuts nothing while cond_2 <= cg <= 1e15
    const bool suspect = fail || !(cg <= 1e15);
    if (pinv_on && m <= SPI_PINV_MAX_M && suspect)
      route[s] = fail ? 4 : 3;
    else
      route[s] = fail ? 2 : 1;
  }
}

// EDK systems whose drift rows are linearly dependent with the
// unbiasedness row (a drift constant over the stations, two proportional
// drifts): F = [1 | drifts] is then rank deficient, the Schur complement
// F'A^-1 F of the Cholesky path singular, and the reference's saddle
// matrix singular, which its pinv resolves. Such systems are sent down the
// exact-inverse path (status = n + 1): F'F's Cholesky with pivots under
// 1e-12 of its diagonal's largest entry marks them (a <= GA rows, one
// thread after the block sums).
__global__ __launch_bounds__(FT) void k_drift_check(spi_domain_t dom, spi_systems_t sys,
                                                   int32_t* __restrict__ status) {
  const int s = blockIdx.x;
  const int a = extra_rows(sys.kind, dom.n_drift);
  if (a < 2 || status[s] != 0) return;
  SysView v = sys_view(sys, s);
  const int n = v.n;
  __shared__ double red[FT / 32];
  __shared__ double M[GA][GA];
  auto fcol = [&](int k, int i) {
    return (k == 0) ? 1.0 : dom.stn_drift[(int64_t)v.idx[i] * dom.n_drift + (k - 1)];
  };
  for (int k = 0; k < a; ++k)
    for (int l = 0; l <= k; ++l) {
      double t = 0.0;
      for (int i = threadIdx.x; i < n; i += FT) t = fma(fcol(k, i), fcol(l, i), t);
      t = block_sum(t, red);
      if (threadIdx.x == 0) M[k][l] = M[l][k] = t;
    }
  __syncthreads();
  if (threadIdx.x == 0) {
    double dmax = 0.0;
    for (int k = 0; k < a; ++k) dmax = fmax(dmax, M[k][k]);
    bool dep = !(dmax > 0.0);
    for (int j = 0; j < a && !dep; ++j) {
      double d = M[j][j];
      for (int c = 0; c < j; ++c) d -= M[j][c] * M[j][c];
      if (!(d > 1e-12 * dmax)) {
        dep = true;
        break;
      }
      const double lj = sqrt(d);
      M[j][j] = lj;
      for (int r = j + 1; r < a; ++r) {
        double t = M[r][j];
        for (int c = 0; c < j; ++c) t -= M[r][c] * M[j][c];
        M[r][j] = t / lj;
      }
    }
    if (dep) status[s] = n + 1;
  }
}

// FP32 copy of every system's matrix (the refinement path's factor).
__global__ void k_to_f32(spi_systems_t sys, const double* __restrict__ l_arena,
                         float* __restrict__ l32) {
  const int s = blockIdx.y;
  SysView v = sys_view(sys, s);
  const int64_t nn = (int64_t)v.n * v.n;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nn;
       e += (int64_t)gridDim.x * blockDim.x)
    l32[v.moff + e] = (float)l_arena[v.moff + e];
}

// Which systems keep the FP32 factor: it succeeded with cond <= cond_ir;
// the others' status is reset for the FP64 factorisation.
__global__ void k_ir_gate(spi_systems_t sys, spi_krige_ws_t ws, double cond_ir) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= sys.n_sys) return;
  const int keep = ws.status[s] == 0 && ws.cond[s] <= cond_ir;
  ws.ir[s] = keep;
  ws.ir_iters[s] = 0;
  if (!keep) ws.status[s] = 0;
}

// Leave-one-out cross-validation residuals of every station of every step
// (closed form): with P11 = A^-1 - G S^-1 G' the top-left block of the
// inverse saddle matrix, z_i - (kriged value at station i from the others)
// = (P11 z)_i / (P11)_ii = w_hat_i / (|Linv[:, i]|^2 - g_i' S^-1 g_i).
// Equal to solving the n leave-one-out systems of the reference's
// formulation one by one (interp/steps.py:170-435 with station i left out)
// whenever its pinv is the inverse. Route-0 systems only; others get NaN.
__global__ __launch_bounds__(FT) void k_loo(spi_domain_t dom, spi_systems_t sys,
                                           spi_krige_ws_t ws, double* __restrict__ resid) {
  const int s = blockIdx.x;
  SysView v = sys_view(sys, s);
  const int n = v.n;
  const bool ok = ws.route[s] == 0;
  const int sk = sys.kind == SPI_KIND_SK;
  const int a = sk ? 0 : extra_rows(sys.kind, dom.n_drift);
  extern __shared__ double dg[];  // [n] diagonal of P11
  const double* X = ws.linv_arena + v.moff;
  const double* G = ws.g_cols + v.off * GA;
  const double* Si = ws.s_inv + (int64_t)s * GA * GA;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    double d = 0.0;
    if (ok) {
      for (int k = i; k < n; ++k) {
        double x = X[(int64_t)k * n + i];
        d += x * x;
      }
      for (int p = 0; p < a; ++p)
        for (int q = 0; q < a; ++q) d -= G[(int64_t)p * n + i] * Si[p * GA + q] * G[(int64_t)q * n + i];
    }
    dg[i] = d;
  }
  __syncthreads();
  for (int64_t si = sys.step_off[s]; si < sys.step_off[s + 1]; ++si) {
    const int64_t vo = sys.val_off[sys.steps[si]];
    for (int i = threadIdx.x; i < n; i += blockDim.x)
      resid[vo + i] = ok ? ws.w_hat[vo + i] / dg[i] : __longlong_as_double(0x7ff8000000000000LL);
  }
}

static size_t gj_smem(int max_n) {
  return (size_t)(max_n + GA) * (2 * sizeof(double) + sizeof(int));
}

int launch_routes(const spi_domain_t& dom, const spi_systems_t& sys, const spi_krige_ws_t& ws,
                  double cond_max, Gate g, cudaStream_t st) {
  const size_t gsm = gj_smem(sys.max_n);
  if (gsm > 200 * 1024) return SPI_ERR_TOO_LARGE;
  if (!smem_opt_in(k_gj, gsm)) return SPI_ERR_CUDA;
  const int pinv_on = ws.pinv_scratch != nullptr;
  k_gj<<<sys.n_sys, FT, gsm, st>>>(dom, sys, ws.l_arena, ws.status, ws.cond, ws.route, cond_max,
                                   pinv_on, g);
  SPI_LAUNCH_CHECK();
  return pinv_on ? launch_pinv(dom, sys, ws, st) : SPI_OK;
}

}  // namespace spi

using namespace spi;



static int check_sys(const spi_domain_t* dom, const spi_systems_t* sys) {
  if (!dom || !sys) return SPI_ERR_ARG;
  if (sys->n_sys < 0 || sys->max_n < 0) return SPI_ERR_ARG;
  if (sys->kind < SPI_KIND_OK || sys->kind > SPI_KIND_EDK) return SPI_ERR_ARG;
  if (dom->n_drift < 0 || dom->n_drift > SPI_MAX_DRIFT) return SPI_ERR_TOO_LARGE;
  if (sys->kind == SPI_KIND_EDK && dom->n_drift > 0 && (!dom->stn_drift || !dom->cell_drift))
    return SPI_ERR_ARG;
  if (sys->n_sys > 65535) return SPI_ERR_TOO_LARGE;
  return SPI_OK;
}

static int check_ws(const spi_krige_ws_t* ws) {
  if (!ws || !ws->l_arena || !ws->status || !ws->route || !ws->cond || !ws->shift ||
      !ws->w_hat || !ws->beta || !ws->g_cols || !ws->s_inv || !ws->g_colsum)
    return SPI_ERR_ARG;
  return SPI_OK;
}

static bool ir_mode(const spi_krige_ws_t* ws) {
  return ws->l32 && !ws->linv_arena && ws->ir && ws->ir_iters;
}

extern "C" int spi_krige_factor(const spi_domain_t* dom, const spi_systems_t* sys,
                                const spi_krige_ws_t* ws, double cond_max,
                                spi_stream_t stream) {
  int rc = check_sys(dom, sys);
  if (rc) return rc;
  if (sys->n_sys == 0) return SPI_OK;
  if ((rc = check_ws(ws))) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  spi_domain_t d = *dom;
  spi_systems_t sy = *sys;
  int64_t nn = (int64_t)sys->max_n * sys->max_n;
  int gx = (int)((nn + 255) / 256);
  if (gx > 64) gx = 64;
  if (gx < 1) gx = 1;
  const bool ir = ir_mode(ws);
  k_build_sys<<<dim3(gx, sys->n_sys), 256, 0, st>>>(d, sy, ws->l_arena, ws->shift, ir ? 1 : 0);
  SPI_LAUNCH_CHECK();
  const Gate every{nullptr, 0}, not_kept{ws->ir, 0};
  if (ir) {
    // FP32 factor first; systems that keep it skip the FP64 one
    k_to_f32<<<dim3(gx, sys->n_sys), 256, 0, st>>>(sy, ws->l_arena, ws->l32);
    if ((rc = launch_chol<float>(sy, ws->l32, ws->status, every, st))) return rc;
    if ((rc = launch_trinv<float>(sy, ws->l32, ws->l32, ws->status, ws->cond, 1, every, st)))
      return rc;
    k_ir_gate<<<(sys->n_sys + 255) / 256, 256, 0, st>>>(sy, *ws,
                                                       ws->cond_ir > 0 ? ws->cond_ir : 1e10);
    SPI_LAUNCH_CHECK();
  }
  const Gate g = ir ? not_kept : every;
  if ((rc = launch_chol<double>(sy, ws->l_arena, ws->status, g, st))) return rc;
  // the inverse factor: an arena of its own where the OK variance reads it
  // (zeros above the diagonal), else over the factor
  double* x = ws->linv_arena ? ws->linv_arena : ws->l_arena;
  if ((rc = launch_trinv<double>(sy, ws->l_arena, x, ws->status, ws->cond,
                                 ws->linv_arena ? 0 : 1, g, st)))
    return rc;
  if (gj_smem(sys->max_n) > 200 * 1024) return SPI_ERR_TOO_LARGE;
  if (sys->kind == SPI_KIND_EDK) {
    k_drift_check<<<sys->n_sys, FT, 0, st>>>(d, sy, ws->status);
    SPI_LAUNCH_CHECK();
  }
  if (ws->pinv_used) {
    if (cudaMemsetAsync(ws->pinv_used, 0, sizeof(int32_t) * (size_t)sys->n_sys, st) !=
        cudaSuccess)
      return SPI_ERR_CUDA;
  }
  if (!ws->gj_scratch) return launch_routes(d, sy, *ws, cond_max, every, st);
  const int pinv_on = ws->pinv_scratch != nullptr;
  if ((rc = launch_gj_multi(d, sy, *ws, cond_max, pinv_on, st))) return rc;
  if (pinv_on) return launch_pinv(d, sy, *ws, st);
  return SPI_OK;
}

extern "C" int spi_krige_duals(const spi_domain_t* dom, const spi_systems_t* sys,
                               const double* vals, const spi_krige_ws_t* ws,
                               spi_stream_t stream) {
  int rc = check_sys(dom, sys);
  if (rc) return rc;
  if (sys->n_sys == 0) return SPI_OK;
  if ((rc = check_ws(ws))) return rc;
  if (!vals) return SPI_ERR_ARG;
  return launch_duals(*dom, *sys, *ws, vals, (cudaStream_t)stream);
}

extern "C" int spi_krige_loo(const spi_domain_t* dom, const spi_systems_t* sys,
                             const spi_krige_ws_t* ws, double* resid, spi_stream_t stream) {
  int rc = check_sys(dom, sys);
  if (rc) return rc;
  if (sys->n_sys == 0) return SPI_OK;
  if ((rc = check_ws(ws))) return rc;
  if (!resid || !ws->linv_arena) return SPI_ERR_ARG;
  size_t smem = (size_t)sys->max_n * sizeof(double);
  if (smem > 200 * 1024) return SPI_ERR_TOO_LARGE;
  if (!smem_opt_in(k_loo, smem)) return SPI_ERR_CUDA;
  k_loo<<<sys->n_sys, FT, smem, (cudaStream_t)stream>>>(*dom, *sys, *ws, resid);
  SPI_LAUNCH_CHECK();
  return SPI_OK;
}
