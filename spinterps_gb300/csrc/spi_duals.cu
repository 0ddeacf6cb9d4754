// The dual vectors of every system of a batch: G = A^-1 F, S = F'G, S^-1,
// 1'G, and per step w_hat = A^-1 z - G beta, beta = S^-1 F'A^-1 z.
//
// A^-1 is applied with the inverse factor Linv (spi_chol.cu) as two products
// with a triangular matrix, rows and columns spread over a cluster of CTAs.
// Substitution with the factor itself, the earlier form, is a chain of n / 32
// dependent blocks on one SM: 244 ms for 8 systems of 2900 stations, 23 ms
// for 8 of 750 (now 6.3 ms and 0.6 ms). Vectors go four at a time, so that a matrix entry is read
// once for four products.
//
// Vectors live in every CTA's shared memory; a product's entry is computed
// by one warp and stored into all CTAs of the cluster at once (lane 8 v + c
// holds vector v and writes it to CTA c), so a cluster barrier separates the
// products and nothing goes through global memory.
//
// Systems that keep an FP32 inverse factor (ws.ir[s] == 1) are refined: the
// correction is computed in FP32 (it only has to be right to a few digits),
// the residual b - A x in FP64 with the full matrix kept in l_arena.
#include <cooperative_groups.h>

#include "spi_factor.cuh"

namespace cg = cooperative_groups;

namespace spi {

namespace {

constexpr int KV = 4;        // vectors per pass
constexpr int DT = 512;      // threads per CTA: the products wait on loads
constexpr int DW = DT / 32;  // warps per CTA
constexpr int RW = 8;        // warps whose partial sums shared memory holds
constexpr int MAXCS = 8;     // CTAs per cluster, at most
constexpr int NSUM = GA * GA + GA + KV * GA;

// Marks a system whose refinement did not converge in ws.ir_iters.
constexpr int kIrFailed = 0x40000000;

// Sums v[0..3] over the warp's lanes; lane 8 k + c returns vector k's sum:
// each exchange halves the number of sums a lane carries (6 additions where
// four butterflies take 20, on a pipe that issues one in 16 cycles).
template <typename T>
__device__ __forceinline__ T reduce4(const T (&v)[KV], int lane) {
  const bool u = lane & 16, w = lane & 8;
  T s0 = u ? v[2] : v[0], s1 = u ? v[3] : v[1];
  const T t0 = u ? v[0] : v[2], t1 = u ? v[1] : v[3];
  s0 += __shfl_xor_sync(0xffffffffu, t0, 16);
  s1 += __shfl_xor_sync(0xffffffffu, t1, 16);
  T r = w ? s1 : s0;
  const T t = w ? s0 : s1;
  r += __shfl_xor_sync(0xffffffffu, t, 8);
  r += __shfl_xor_sync(0xffffffffu, r, 4);
  r += __shfl_xor_sync(0xffffffffu, r, 2);
  r += __shfl_xor_sync(0xffffffffu, r, 1);
  return r;
}

// |x| as a float from the double's high word (20 significant bits, no
// conversion on the FP64 pipe); 0 under float's range.
__device__ __forceinline__ float abs_hi(double x) {
  const int h = (__double2hiint(x) & 0x7fffffff) - (896 << 20);
  return h <= 0 ? 0.f : __int_as_float(min(h, 0x0fefffff) << 3);
}

// S^-1 of the small a x a Schur complement by Gauss-Jordan with partial
// pivoting (one thread), zero-padded.
__device__ void schur_inverse(const double (*S)[GA], int a, double (*Si)[GA]) {
  double M[GA][2 * GA];
  for (int i = 0; i < a; ++i)
    for (int j = 0; j < 2 * a; ++j) M[i][j] = (j < a) ? S[i][j] : (j - a == i ? 1.0 : 0.0);
  for (int c = 0; c < a; ++c) {
    int p = c;
    for (int r = c + 1; r < a; ++r)
      if (fabs(M[r][c]) > fabs(M[p][c])) p = r;
    if (p != c)
      for (int j = 0; j < 2 * a; ++j) {
        const double t = M[c][j];
        M[c][j] = M[p][j];
        M[p][j] = t;
      }
    const double piv = M[c][c];
    for (int j = 0; j < 2 * a; ++j) M[c][j] /= piv;
    for (int r = 0; r < a; ++r)
      if (r != c) {
        const double f = M[r][c];
        for (int j = 0; j < 2 * a; ++j) M[r][j] -= f * M[c][j];
      }
  }
  for (int i = 0; i < GA; ++i)
    for (int j = 0; j < GA; ++j) Si[i][j] = (i < a && j < a) ? M[i][a + j] : 0.0;
}

enum Phase { kAll, kSolve, kSteps };

struct Cta {
  cg::cluster_group cl;
  int cs, rank, lane, warp;
};

// First row this CTA owns of its local block lb (blocks of 32 rows are dealt
// to the cluster's CTAs in turn).
__device__ __forceinline__ int own_row(const Cta& c, int lb) { return (c.rank + c.cs * lb) * 32; }

// y = X v for the pass's vectors (X lower triangular), stored into yb of
// every CTA of the cluster.
template <typename TX, typename TV>
__device__ void lower_product(const Cta& c, const TX* __restrict__ X, int n, int nk, const TV* v,
                              TV* y, double* base) {
  const int nw = c.cs * DW;
  // this thread's copy of y in the CTA it writes to
  const int tc = c.lane & 7;
  double* rb = c.cl.map_shared_rank(base, tc < c.cs ? tc : 0);
  TV* yr = reinterpret_cast<TV*>(rb) + (y - reinterpret_cast<TV*>(base));
  for (int i = c.rank * DW + c.warp; i < n; i += nw) {
    const TX* row = X + (int64_t)i * n;
    TV acc[KV] = {};
#pragma unroll 4
    for (int j = c.lane; j <= i; j += 32) {
      const TV x = (TV)row[j];
#pragma unroll
      for (int k = 0; k < KV; ++k)
        if (k < nk) acc[k] += x * v[k * n + j];
    }
    const TV r = reduce4(acc, c.lane);
    if (tc < c.cs && (c.lane >> 3) < nk) yr[(c.lane >> 3) * n + i] = r;
  }
}

// z = X' y for the pass's vectors on the rows this CTA owns; fin(k, i, z) is
// called once per vector and owned row.
template <typename TX, typename TV, typename F>
__device__ void lower_t_product(const Cta& c, const TX* __restrict__ X, int n, int nk,
                                const TV* y, double* red_, F fin) {
  TV* red = reinterpret_cast<TV*>(red_);  // [RW][KV][32]
  for (int lb = 0;; ++lb) {
    const int j0 = own_row(c, lb);
    if (j0 >= n) break;
    const int j = j0 + c.lane;
    TV acc[KV] = {};
    if (j < n) {
#pragma unroll 4
      for (int i = j0 + c.warp; i < n; i += DW) {
        // (above the diagonal X is scratch)
        const TV x = i >= j ? (TV)X[(int64_t)i * n + j] : TV(0);
#pragma unroll
        for (int k = 0; k < KV; ++k)
          if (k < nk) acc[k] += x * y[k * n + i];
      }
    }
    __syncthreads();
    if (c.warp >= RW)
#pragma unroll
      for (int k = 0; k < KV; ++k) red[((c.warp - RW) * KV + k) * 32 + c.lane] = acc[k];
    __syncthreads();
    if (c.warp < RW)
#pragma unroll
      for (int k = 0; k < KV; ++k) red[(c.warp * KV + k) * 32 + c.lane] += acc[k];
    __syncthreads();
    if (threadIdx.x < KV * 32) {
      const int k = threadIdx.x >> 5;
      TV t = TV(0);
#pragma unroll
      for (int w = 0; w < RW; ++w) t += red[(w * KV + k) * 32 + c.lane];
      if (j < n && k < nk) fin(k, j, lb, t);
    }
  }
  __syncthreads();
}

__global__ __launch_bounds__(DT) void k_duals(spi_domain_t dom, spi_systems_t sys,
                                             spi_krige_ws_t ws, const double* __restrict__ vals,
                                             int phase, int fallback, int nk, int max_n,
                                             int cap) {
  Cta c{cg::this_cluster(), 0, 0, (int)(threadIdx.x & 31), (int)(threadIdx.x >> 5)};
  c.cs = c.cl.num_blocks();
  c.rank = c.cl.block_rank();
  const int s = blockIdx.y, gi = blockIdx.x / c.cs, ngrp = gridDim.x / c.cs;
  const int route = ws.route[s];
  // every early return below is the same for the whole cluster
  if (route == 2) return;
  const bool linv = ws.linv_arena != nullptr;
  // (in the fallback pass kSolve also takes what has left the Cholesky path)
  if (phase == kAll ? (route == 0 && !linv)
                    : route != 0 && !(fallback && phase == kSolve && route == 1))
    return;
  if (fallback && ws.ir[s] != 2) return;
  const SysView v = sys_view(sys, s);
  const int n = v.n, tid = threadIdx.x;
  const int sk = sys.kind == SPI_KIND_SK;
  const int a = sk ? 1 : extra_rows(sys.kind, dom.n_drift);
  const int64_t sb = sys.step_off[s];
  const int nsteps = (int)(sys.step_off[s + 1] - sb);
  // this cluster's steps: at least what fits beside F in its first pass
  const bool with_f = phase != kSteps;
  const int beside = with_f ? max(1, nk - a) : nk;
  // (kSolve: one cluster per system takes the first steps; kSteps: the rest)
  const int first = phase == kSteps ? max(1, nk - a) : 0;
  const int todo =
      phase == kSolve && route == 0 ? min(nsteps, beside) : max(0, nsteps - first);
  const int per = max(beside, (todo + ngrp - 1) / ngrp);
  const int q0 = min(todo, gi * per) + first, q1 = min(todo, (gi + 1) * per) + first;
  if (gi > 0 ? q0 >= q1 : (!with_f && q0 >= q1)) return;

  // xa: the vectors of the pass (with refinement the solution x); yb: the
  // gathered first product (with refinement two float arrays, residual and
  // product); own: results of the rows this CTA owns [a + nk][cap]
  extern __shared__ double sm[];
  double* xa = sm;                        // [nk][n]
  double* yb = sm + (int64_t)nk * max_n;  // [nk][n]
  double* own = sm + (int64_t)2 * nk * max_n;
  __shared__ double red[RW * KV * 32];
  static_assert(DW == 2 * RW, "two warps per partial sum");
  __shared__ double part[MAXCS][NSUM];
  __shared__ float bem[2][MAXCS];
  __shared__ double S[GA][GA], Si[GA][GA], colsum[GA], bt[KV][GA];
  __shared__ double scale[KV], iscale[KV];
  __shared__ double wred[DW];
  double* G = ws.g_cols + v.off * GA;  // column k at G + k * n
  auto fcol = [&](int k, int i) {
    return (k == 0) ? 1.0 : dom.stn_drift[(int64_t)v.idx[i] * dom.n_drift + (k - 1)];
  };
  auto step_vals = [&](int q) { return vals + sys.val_off[sys.steps[sb + q]]; };

  if (route == 1) {
    // the inverse saddle matrix P (m x m): G = P 1, w_hat = P z, a warp per
    // row of the cluster; vector 0 of group 0's first pass is 1
    const int ar = sk ? 0 : a, m = n + ar;
    const double* P = ws.l_arena + v.moff;
    const int nw = c.cs * DW;
    int q = q0;
    for (bool f = gi == 0; f || q < q1;) {
      const int lead = f ? 1 : 0, ns = min(nk - lead, q1 - q);
      __syncthreads();
      for (int k = 0; k < lead + ns; ++k) {
        const double* z = k < lead ? nullptr : step_vals(q + k - lead);
        for (int i = tid; i < n; i += DT) xa[k * n + i] = z ? z[i] : 1.0;
      }
      __syncthreads();
      for (int i = c.rank * DW + c.warp; i < m; i += nw) {
        const double* row = P + (int64_t)i * m;
        double acc[KV] = {};
#pragma unroll 4
        for (int j = c.lane; j < n; j += 32) {
          const double x = row[j];
#pragma unroll
          for (int k = 0; k < KV; ++k)
            if (k < lead + ns) acc[k] = fma(x, xa[k * n + j], acc[k]);
        }
        const double r = reduce4(acc, c.lane);
        const int k = c.lane >> 3;
        if ((c.lane & 7) == 0 && k < lead + ns) {
          if (k < lead) {
            if (i < n) {
              G[i] = r;
              // SK: |u| as a second column (the FP32 tier's bound of its
              // sum check's rounding)
              if (sk) G[n + i] = fabs(r);
            } else {
              ws.g_colsum[(int64_t)s * GA + (i - n)] = r;
            }
          } else {
            const int j = sys.steps[sb + q + k - lead];
            if (i < n) ws.w_hat[sys.val_off[j] + i] = r;
            else ws.beta[(int64_t)j * GA + (i - n)] = r;
          }
        }
      }
      if (c.rank == 0 && tid >= ar && tid < GA) {
        if (f) ws.g_colsum[(int64_t)s * GA + tid] = 0.0;
        for (int k = 0; k < ns; ++k) ws.beta[(int64_t)sys.steps[sb + q + k] * GA + tid] = 0.0;
      }
      q += ns;
      f = false;
    }
    return;
  }

  const bool ir = !linv && ws.l32 && ws.ir && ws.ir[s] == 1;
  const double* X64 = (linv ? ws.linv_arena : ws.l_arena) + v.moff;
  const float* X32 = ir ? ws.l32 + v.moff : nullptr;
  const double* A = ws.l_arena + v.moff;
  float* rf = reinterpret_cast<float*>(yb);  // residual [nk][n]
  float* yf = rf + nk * n;                   // FP32 product [nk][n]
  double* base = sm;

  // A^-1 applied to nv vectors, entry i of vector k given by bval(k, i); the
  // owned rows of vector k go to own[(slot + k) * cap + ...]
  auto solve = [&](int nv, int slot, auto bval) {
    if (!ir) {
      __syncthreads();
      for (int e = tid; e < nk * n; e += DT) {
        const int k = e / n;
        xa[e] = k < nv ? bval(k, e - k * n) : 0.0;
      }
      c.cl.sync();  // every CTA of the cluster runs, its yb free
      lower_product<double, double>(c, X64, n, nk, xa, yb, base);
      c.cl.sync();
      lower_t_product<double, double>(c, X64, n, nk, yb, red, [&](int k, int i, int lb, double z) {
        if (k < nv) own[(slot + k) * cap + lb * 32 + (i & 31)] = z;
      });
      c.cl.sync();  // yb is free again
      return;
    }
    // each vector scaled by a power of two to at most 1, so that FP32 holds
    // its residuals whatever the values' unit
    for (int k = 0; k < nk; ++k) {
      double t = 0.0;
      if (k < nv)
        for (int i = tid; i < n; i += DT) t = fmax(t, fabs(bval(k, i)));
      for (int o = 16; o > 0; o >>= 1) t = fmax(t, __shfl_xor_sync(0xffffffffu, t, o));
      __syncthreads();
      if (c.lane == 0) wred[c.warp] = t;
      __syncthreads();
      if (tid == 0) {
        for (int w = 1; w < DW; ++w) t = fmax(t, wred[w]);
        int e = 0;
        if (t > 0.0 && t < 1e300) frexp(t, &e);
        scale[k] = ldexp(1.0, e);
        iscale[k] = ldexp(1.0, -e);
      }
    }
    __syncthreads();
    for (int e = tid; e < nk * n; e += DT) {
      const int k = e / n;
      xa[e] = 0.0;
      rf[e] = k < nv ? (float)(bval(k, e - k * n) * iscale[k]) : 0.f;
    }
    c.cl.sync();
    const double tol = sqrt((double)n) * 2.220446049250313e-16;
    float prev = __int_as_float(0x7f800000);
    bool conv = false;
    int it = 0;
    for (;; ++it) {
      // x += Linv' Linv r, in FP32
      lower_product<float, float>(c, X32, n, nk, rf, yf, base);
      c.cl.sync();
      lower_t_product<float, float>(c, X32, n, nk, yf, red, [&](int k, int i, int lb, float z) {
        const double x = xa[k * n + i] + (double)z;
        for (int t = 0; t < c.cs; ++t) c.cl.map_shared_rank(xa, t)[k * n + i] = x;
      });
      c.cl.sync();
      // r = b - A x and the componentwise backward error
      float be = 0.f;
      const int tc = c.lane & 7, kk = c.lane >> 3;
      float* rr = reinterpret_cast<float*>(c.cl.map_shared_rank(base, tc < c.cs ? tc : 0)) +
                  (rf - reinterpret_cast<float*>(base));
      for (int i = c.rank * DW + c.warp; i < n; i += c.cs * DW) {
        const double* row = A + (int64_t)i * n;
        double t[KV] = {};
        float ta[KV] = {};
#pragma unroll 4
        for (int j = c.lane; j < n; j += 32) {
          const double x = row[j];
          const float xf = abs_hi(x);
#pragma unroll
          for (int k = 0; k < KV; ++k)
            if (k < nv) {
              const double y = xa[k * n + j];
              t[k] = fma(x, y, t[k]);
              ta[k] = fmaf(xf, abs_hi(y), ta[k]);
            }
        }
        const double tt = reduce4(t, c.lane);
        const float tb = reduce4(ta, c.lane);
        float r = 0.f;
        if (kk < nv) {
          const double b = bval(kk, i) * iscale[kk];
          r = (float)(b - tt);
          const float den = tb + fabsf((float)b);
          if (den > 0.f) be = fmaxf(be, fabsf(r) / den);
          else if (r != 0.f) be = __int_as_float(0x7f800000);
          if (r != r) be = __int_as_float(0x7f800000);
        }
        if (tc < c.cs && kk < nk) rr[kk * n + i] = r;
      }
      for (int o = 16; o > 0; o >>= 1) be = fmaxf(be, __shfl_xor_sync(0xffffffffu, be, o));
      __syncthreads();
      if (c.lane == 0) wred[c.warp] = (double)be;
      __syncthreads();
      if (tid < c.cs) {
        double m = 0.0;
        for (int w = 0; w < DW; ++w) m = fmax(m, wred[w]);
        c.cl.map_shared_rank(&bem[0][0], tid)[(it & 1) * MAXCS + c.rank] = (float)m;
      }
      c.cl.sync();
      be = 0.f;
      for (int w = 0; w < c.cs; ++w) be = fmaxf(be, bem[it & 1][w]);
      if ((double)be <= tol) {
        conv = true;
        break;
      }
      // a factor too far from A makes no progress: stop once a correction
      // fails to halve the backward error
      if (it == SPI_IR_MAX_ITERS || !(be < 0.5f * prev)) break;
      prev = be;
    }
    for (int lb = 0;; ++lb) {
      const int j0 = own_row(c, lb);
      if (j0 >= n) break;
      for (int e = tid; e < nv * 32; e += DT) {
        const int k = e >> 5, i = j0 + (e & 31);
        if (i < n) own[(slot + k) * cap + lb * 32 + (e & 31)] = xa[k * n + i] * scale[k];
      }
    }
    if (c.rank == 0 && tid == 0 && ws.ir_iters) {
      atomicMax(ws.ir_iters + s, it);
      if (!conv) atomicOr(ws.ir_iters + s, kIrFailed);
    }
    c.cl.sync();
  };

  // sums over the system's rows, number by number: every CTA its owned rows,
  // all of them gathered in every CTA
  auto gather_sums = [&](int cnt, auto term) {
    __syncthreads();
    for (int q = c.warp; q < cnt; q += DW) {
      double t = 0.0;
      for (int lb = 0;; ++lb) {
        const int i = own_row(c, lb) + c.lane;
        if (own_row(c, lb) >= n) break;
        if (i < n) t += term(q, i, lb * 32 + c.lane);
      }
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (c.lane < c.cs) c.cl.map_shared_rank(&part[0][0], c.lane)[c.rank * NSUM + q] = t;
    }
    c.cl.sync();
  };
  auto total = [&](int q) {
    double t = 0.0;
    for (int w = 0; w < c.cs; ++w) t += part[w][q];
    return t;
  };
  // the steps q .. q + ns - 1, whose A^-1 z are in own slots a ..
  auto finish_steps = [&](int q, int ns) {
    if (!sk) {
      gather_sums(ns * a, [&](int e, int i, int o) {
        return fcol(e % a, i) * own[(a + e / a) * cap + o];
      });
      for (int e = tid; e < ns * GA; e += DT) {
        const int k = e / GA, m = e % GA;
        double t = 0.0;
        if (m < a)
          for (int l = 0; l < a; ++l) t += Si[m][l] * total(k * a + l);
        bt[k][m] = t;
      }
    } else {
      for (int e = tid; e < ns * GA; e += DT) bt[e / GA][e % GA] = 0.0;
    }
    __syncthreads();
    for (int lb = 0;; ++lb) {
      const int j0 = own_row(c, lb);
      if (j0 >= n) break;
      for (int e = tid; e < ns * 32; e += DT) {
        const int k = e >> 5, i = j0 + (e & 31), o = lb * 32 + (e & 31);
        if (i >= n) continue;
        double w = own[(a + k) * cap + o];
        if (!sk)
          for (int m = 0; m < a; ++m)
            w -= (with_f ? own[m * cap + o] : G[(int64_t)m * n + i]) * bt[k][m];
        ws.w_hat[sys.val_off[sys.steps[sb + q + k]] + i] = w;
      }
    }
    if (c.rank == 0)
      for (int e = tid; e < ns * GA; e += DT)
        ws.beta[(int64_t)sys.steps[sb + q + e / GA] * GA + e % GA] = bt[e / GA][e % GA];
    c.cl.sync();  // part and bt are free again
  };

  int q = q0;
  if (with_f) {
    int ns0 = 0;  // steps solved beside the last columns of F
    for (int k0 = 0; k0 < a; k0 += nk) {
      const int kf = min(nk, a - k0);
      ns0 = (k0 + nk >= a) ? min(nk - kf, q1 - q0) : 0;
      solve(kf + ns0, k0, [&](int k, int i) {
        return k < kf ? fcol(k0 + k, i) : step_vals(q0 + k - kf)[i];
      });
    }
    __syncthreads();
    gather_sums(a * a + a, [&](int e, int i, int o) {
      return e < a * a ? fcol(e / a, i) * own[(e % a) * cap + o] : own[(e - a * a) * cap + o];
    });
    for (int e = tid; e < a * a; e += DT) S[e / a][e % a] = total(e);
    if (tid < GA) colsum[tid] = tid < a ? total(a * a + tid) : 0.0;
    __syncthreads();
    if (tid == 0) schur_inverse(S, a, Si);
    __syncthreads();
    if (gi == 0) {
      if (c.rank == 0) {
        for (int e = tid; e < GA * GA; e += DT)
          ws.s_inv[(int64_t)s * GA * GA + e] = Si[e / GA][e % GA];
        if (tid < GA) ws.g_colsum[(int64_t)s * GA + tid] = colsum[tid];
      }
      for (int lb = 0;; ++lb) {
        const int j0 = own_row(c, lb);
        if (j0 >= n) break;
        for (int e = tid; e < a * 32; e += DT) {
          const int k = e >> 5, i = j0 + (e & 31);
          if (i >= n) continue;
          const double g = own[k * cap + lb * 32 + (e & 31)];
          G[(int64_t)k * n + i] = g;
          // SK: |u| (u = A^-1 1) as a second column: the FP32 cell kernels
          // contract it to bound the rounding of sum(lambda) = u'c
          if (sk) G[n + i] = fabs(g);
        }
      }
    }
    c.cl.sync();  // part is free again
    if (ns0) finish_steps(q0, ns0);
    q += ns0;
  } else {
    for (int e = tid; e < GA * GA; e += DT)
      Si[e / GA][e % GA] = ws.s_inv[(int64_t)s * GA * GA + e];
    __syncthreads();
  }
  for (; q < q1; q += nk) {
    const int ns = min(nk, q1 - q);
    solve(ns, a, [&](int k, int i) { return step_vals(q + k)[i]; });
    __syncthreads();
    finish_steps(q, ns);
  }
}

// Systems whose refinement did not converge fall back to the FP64 factor
// (ir = 2): they are then factored, given their route and solved again. (An
// FP32 factor of a singular matrix, of two gauges in one place for instance,
// has a small pivot of rounding where the FP64 one fails or is far too ill
// conditioned for the Cholesky path.)
constexpr double kFallbackCondMax = 1e13;  // the callers' usual cond_max
__global__ void k_ir_fail_gate(spi_systems_t sys, spi_krige_ws_t ws) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= sys.n_sys) return;
  if (ws.ir[s] == 1 && (ws.ir_iters[s] & kIrFailed)) ws.ir[s] = 2;
}

}  // namespace

int launch_duals(const spi_domain_t& dom, const spi_systems_t& sys, const spi_krige_ws_t& ws,
                 const double* vals, cudaStream_t st) {
  const int n = sys.max_n;
  const int a = sys.kind == SPI_KIND_SK ? 1 : extra_rows(sys.kind, dom.n_drift);
  // CTAs per cluster: the products of small systems are over before a
  // cluster barrier pays
  const int cs = n <= 96 ? 1 : (n <= 256 ? 4 : MAXCS);
  const int cap = ((n + 31) / 32 + cs - 1) / cs * 32;
  // vectors per pass within the shared memory
  int nk = KV;
  auto bytes = [&](int k) {
    return sizeof(double) * ((size_t)2 * k * n + (size_t)(a + k) * cap);
  };
  while (nk > 1 && bytes(nk) > 200 * 1024) --nk;
  if (bytes(nk) > 216000) return SPI_ERR_TOO_LARGE;  // (16 KB are static)
  if (!smem_opt_in(k_duals, bytes(nk))) return SPI_ERR_CUDA;
  auto launch = [&](int phase, int fallback, int groups) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(groups * cs), (unsigned)sys.n_sys);
    cfg.blockDim = dim3(DT);
    cfg.dynamicSmemBytes = bytes(nk);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)cs;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_duals, dom, sys, ws, vals, phase, fallback, nk, n, cap);
  };
  // step groups: enough clusters for the GPU twice over
  int gx = (304 + sys.n_sys * cs - 1) / (sys.n_sys * cs);
  gx = gx > 64 ? 64 : gx;
  cudaError_t e = launch(kAll, 0, gx);
  if (!ws.linv_arena) {
    const bool ir = ws.l32 && ws.ir && ws.ir_iters;
    for (int pass = 0; pass < (ir ? 2 : 1); ++pass) {
      if (pass == 1) {
        k_ir_fail_gate<<<(sys.n_sys + 255) / 256, 256, 0, st>>>(sys, ws);
        const Gate g{ws.ir, 2};
        int rc = launch_chol<double>(sys, ws.l_arena, ws.status, g, st);
        if (rc) return rc;
        if ((rc = launch_trinv<double>(sys, ws.l_arena, ws.l_arena, ws.status, ws.cond, 1, g, st)))
          return rc;
        if ((rc = launch_routes(dom, sys, ws, kFallbackCondMax, g, st))) return rc;
      }
      if (e == cudaSuccess) e = launch(kSolve, pass, 1);
      if (e == cudaSuccess) e = launch(kSteps, pass, gx);
    }
  }
  if (e != cudaSuccess) {
    record_cuda_error(e);
    return SPI_ERR_CUDA;
  }
  SPI_LAUNCH_CHECK();
  return SPI_OK;
}

}  // namespace spi
