// Kriging estimates over all cells for systems too large for the
// shared-memory right-hand side of k_krige_cells (n stations x a cell tile
// beyond 227 KB: n > ~1600 in FP64, ~3500 in FP32), e.g. thousands of
// stations with external drifts. Estimates only: the right-hand side of a
// cell is used once per pass, so it is generated on the fly, never stored.
//
// Layout: one CTA = 8 warps over 32 cells (FP64) or 64 (FP32 tier, two to a
// lane). The 8 warps split the system's stations (warp w takes stations w,
// w + 8, ...). Each lane generates its cells' entries for the warp's station
// (station data are warp-uniform broadcast loads) and accumulates them
// against up to 4 vectors: the system's dual columns (Lagrange / drift rows,
// for the sum check of interp/steps.py:419) and the steps' dual weights. The
// 8 partial sums per cell are reduced in shared memory; more steps than fit
// in one pass regenerate the right-hand side. Precision as k_krige_cells:
// FP64 throughout, or (the mixed path's FP32 tier) double-float entries
// against FP32 hi/lo vector pairs, accumulated in double-float and flushed
// to FP64 every 256 terms: the estimate's error is sum_i dc_i w_i, which
// large dual weights amplify. With ws.cell_yy (the tensor-core |Linv c|^2)
// the FP32 tier also writes the OK variance.
//
// The FP32 tier is bound by the instructions of an entry: about 165 as
// normalised double-floats (rhs_df_single's sqrt, exp and products), about 80
// as the pairs of rho_pair, which are no further from exact (rms 2^-44 of
// the sill for Exp and Gau instead of 2^-41.5, 2^-45 both for Sph and Lin).
// One cell to a lane and 16 warps to an SM left every second issue slot
// empty, waiting on the chain of one entry: two cells to a lane, 32 warps
// (the FP64 totals in shared memory, the entries without a pair form out of
// line), one branch for both cells' cuts, which leaves the inner loop for the
// exact form, and the usual passes' vectors known at compile time. 8 systems
// of 2900 stations, 10^6 cells, 4 vectors: 203 ms as double-floats, 90 with
// the pairs, 72.5 with 32 warps, 66.5 with the exact form outside the loop
// (85% of the issue slots used before that, 109 instructions an entry, some
// of them spills); 8 of 750 stations, 250 000 cells: 33, 19.4, 17.4, 17.0
// ms. (Three CTAs of 80 registers take 6% longer on large grids, a fifth on
// small systems.)
#include <type_traits>

#include "spi_cells.cuh"
#include "spi_rhs.cuh"

namespace spi {

constexpr int STC = 32;  // cells per CTA and cell of a lane
constexpr int SC4 = 2;   // cells of a lane in the FP32 tier
constexpr int SNW = 8;   // warps per CTA (station groups)
constexpr int SSV = 4;   // vectors per pass
constexpr int SCH = 256; // stations per shared-memory chunk (FP32 tier)

// An entry without a pair form (rhs_df_d2); out of line, so that its FP64
// models don't set the registers of the loop below.
inline __device__ __noinline__ df stream_general(const CellsArgs& A, const spi_vg_t* vgp,
                                                 const RhsDf& kd, int sk, double sh, df d2,
                                                 int64_t gc, const int32_t* stp) {
  return rhs_df_d2(A.dom, vgp, kd, sk, sh, d2, gc, stp);
}
// The coordinates up to which squared distances stay within FP32.
constexpr float kFar = 1e18f;

// One shared-memory chunk of stations against the pass's vectors (FP32
// tier): double-float entries times hi/lo vector pairs, the product's head
// by the FMA error, the cross terms, TwoSum into a double-float partial that
// the caller flushes to FP64 every 256 terms. The first np vectors, dual
// columns that feed only the sum check, take a plain FP32 product. A lane's
// two cells share the loads, and their chains overlap.
// CODE: the single structure's model (rho_pair, in units of its sill), or -1.
// SK's entries at or below the cut are zero, OK's / EDK's past it the whole
// sill; entries near it take the exact form (rho_cut), for which the warp
// leaves the inner loop: a call inside it would hold the loop's registers to
// those a call preserves. NP, NV: np and nv
// where they are known at compile time, or -1.
template <int CODE, bool SK, bool TRACK, int NP, int NV>
__device__ __forceinline__ void stream_chunk(const CellsArgs& A, const spi_vg_t* vgp,
                                             const RhsDf& kd, const RhsOne& ko,
                                             const float2* tab, double sh, const float4 (&cp)[2],
                                             const int64_t (&gc)[2], const int32_t* idxc,
                                             const float4* s_sp, const float2 (*s_w)[SSV],
                                             int nj, int warp, int np, int nv,
                                             float (&ph)[SSV][2], float (&pl)[SSV][2],
                                             NearDf (&nf)[2], int j0, float esp) {
  const float lo = ko.lo, hi = ko.hi;
  if constexpr (NV >= 0) np = NP, nv = NV;
  // an entry pair against the vectors
  auto take = [&](const df (&c)[2], int jj) {
#pragma unroll
    for (int v = 0; v < SSV; ++v) {
      if (v >= nv) continue;
      const float2 w = s_w[jj][v];
      if (v < np) {
#pragma unroll
        for (int u = 0; u < 2; ++u) ph[v][u] = __fmaf_rn(c[u].h, w.x, ph[v][u]);
      } else {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const float p = __fmul_rn(c[u].h, w.x);
          float e = __fmaf_rn(c[u].h, w.x, -p);
          e = __fmaf_rn(c[u].h, w.y, e);
          e = __fmaf_rn(c[u].l, w.x, e);
          const df s2 = two_sum(ph[v][u], p);
          ph[v][u] = s2.h;
          pl[v][u] += s2.l + e;
        }
      }
    }
  };
  if constexpr (CODE < 0) {
    for (int jj = warp; jj < nj; jj += SNW) {
      df c[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const df d2 = df_dist2(cp[u], s_sp[jj]);
        if constexpr (TRACK) nf[u].add(d2, j0 + jj, esp);
        c[u] = stream_general(A, vgp, kd, SK, sh, d2, gc[u], idxc + jj);
      }
      take(c, jj);
    }
  } else {
    int jj = warp;
    while (jj < nj) {
      df c[2];
      bool cut = false;
      for (; jj < nj; jj += SNW) {
        const float4 sp = s_sp[jj];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const df s = dist2_pair(cp[u], sp);
          if constexpr (TRACK) nf[u].add(s, j0 + jj, esp);
          c[u] = rho_pair<CODE>(ko, s, tab);
          if constexpr (SK) {
            const bool z = c[u].h < lo;
            c[u].h = z ? 0.f : c[u].h;
            c[u].l = z ? 0.f : c[u].l;
          }
        }
        // (one branch for both cells, and out of the loop for the exact form)
        cut = SK ? (c[0].h >= lo && c[0].h <= hi) || (c[1].h >= lo && c[1].h <= hi)
                 : fmaxf(c[0].h, c[1].h) >= hi;
        if (__any_sync(0xffffffffu, cut)) break;
        take(c, jj);
      }
      if (jj < nj) {
#pragma unroll
        for (int u = 0; u < 2; ++u)
          if (SK ? c[u].h >= lo && c[u].h <= hi : c[u].h >= hi)
            c[u] = rho_cut(A.dom, vgp, kd, ko, SK, sh, gc[u], idxc + jj, c[u]);
        take(c, jj);
        jj += SNW;
      }
    }
  }
}

template <typename T, typename OutT>
__global__ __launch_bounds__(STC * SNW, sizeof(T) == 4 ? 4 : 2) void k_krige_cells_stream(
    CellsArgs A) {
  constexpr int NC = sizeof(T) == 4 ? SC4 : 1;  // cells of a lane
  constexpr int TC = STC * NC;                  // cells of the CTA
  const int s = blockIdx.y;
  const int64_t C = A.dom.n_cells;
  const int64_t c0 = (int64_t)blockIdx.x * TC;
  if (c0 >= C || A.done.has(s)) return;
  const int route = A.ws.route[s];
  {
    const bool fast = fp32_tier(A.ws, s, A.cond_split, A.sys.kind == SPI_KIND_SK);
    if ((A.route_filter == 1 && !fast) || (A.route_filter == 2 && fast)) return;
  }
  const bool prim = route == 1;
  const bool failed = route == 2;
  const int64_t soff = A.sys.stn_off[s];
  const int n = (int)(A.sys.stn_off[s + 1] - soff);
  const int32_t* idx = A.sys.stn_idx + soff;
  const int sk = A.sys.kind == SPI_KIND_SK;
  const int a = sk ? 1 : extra_rows(A.sys.kind, A.dom.n_drift);
  // (SK in an FP32 tier adds |u|, the bound of its sum check's rounding,
  // on either route)
  const int ndual = (sk && sizeof(T) == 4) ? 2 : (prim ? 1 : a);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t st0 = A.sys.step_off[s];
  const int nsteps = (int)(A.sys.step_off[s + 1] - st0);
  const int nvec = ndual + nsteps;
  // OK / EDK without the variance: the dual columns feed only the sum
  // check, and sum(lambda) = q0 - sum_k S_0k nu_k is 1 identically whatever
  // q is (nu = S^-1 (q - f)); they need no more than FP32 (the estimates,
  // SK's u'c and the OK variance's q0 keep double-float)
  const bool var_needed = A.want_var && A.out.var != nullptr && !sk;
  const int plain_duals = (sizeof(T) == 4 && !sk && !prim && !var_needed) ? ndual : 0;
  const spi_vg_t vg = A.sys.vg[s];
  const double sh = A.ws.shift[s];

  __shared__ double red[SNW][SSV][TC];
  __shared__ double vres[SSV][TC];
  __shared__ double qsh[GA][TC];  // dual columns (more than a pass holds: EDK, 4 drifts on)
  __shared__ int okf[TC], nnb[TC];
  __shared__ double cvar[TC];
  __shared__ const double* vp64[SSV];
  __shared__ const float* vph[SSV];
  __shared__ const float* vpl[SSV];
  __shared__ int any_bad;
  __shared__ int any_chk;
  __shared__ float4 s_sp[sizeof(T) == 4 ? SCH : 1];
  __shared__ __align__(16) float2 s_w[sizeof(T) == 4 ? SCH : 1][SSV];
  __shared__ float2 s_tab[sizeof(T) == 4 ? 256 : 1];
  // the FP32 tier's nearest-station candidates per station group (warp)
  // and cell, from the first pass's right-hand sides (written over red once
  // the pass's sums are reduced), and the cells they leave ambiguous
  NearDf* s_nf = reinterpret_cast<NearDf*>(&red[0][0][0]);
  static_assert(sizeof(NearDf) * SNW * TC <= sizeof(red), "candidates fit in red");
  __shared__ int namb[TC];
  const bool fuse_nnb = sizeof(T) == 4 && A.dom.split_res > 0.0;
  const float esp = (float)(A.dom.split_res * 0x1p-24);
  bool nf_ready = false;

  // this lane's cells c0 + lane, c0 + lane + 32 (past the grid: its last)
  int64_t gc[NC];
#pragma unroll
  for (int u = 0; u < NC; ++u) {
    gc[u] = c0 + u * STC + lane;
    if (gc[u] >= C) gc[u] = C - 1;
  }
  OutT* est_out = reinterpret_cast<OutT*>(A.out.est);
  // the OK variance needs |Linv c|^2 per cell from the tensor-core kernel
  const bool var_out = sizeof(T) == 4 && A.want_var && A.out.var != nullptr && !sk &&
                       A.ws.cell_yy != nullptr;
  OutT* var_outp = reinterpret_cast<OutT*>(A.out.var);
  auto emit = [&](int cell, int vstep, double accv) {
    const int64_t g = c0 + cell;
    if (g >= C) return;
    const int j = A.sys.steps[st0 + vstep];
    const int64_t row = A.sys.out_row[j];
    double e;
    if (okf[cell]) {
      e = accv;
      if (!sk) {
        const double* bt = A.ws.beta + (int64_t)j * GA;
        e += bt[0];
        for (int k = 1; k < a; ++k) e += bt[k] * A.dom.cell_drift[(int64_t)(k - 1) * C + g];
      }
    } else {
      e = A.vals[A.sys.val_off[j] + nnb[cell]];
    }
    est_out[row * C + g] = cast_out<OutT>(clip_est(e, A.out));
    if (var_out) var_outp[row * C + g] = cast_out<OutT>(okf[cell] ? cvar[cell] : 0.0);
  };
  // the nearest station of every cell that failed the sum check: from the
  // right-hand sides' squared distances where they decide it, else (and
  // without them) the exact FP64 search
  auto nearest = [&]() {
    __syncthreads();
    if (any_bad) {
      if (tid < TC) {
        int amb = 1;
        if constexpr (sizeof(T) == 4) {
          if (nf_ready) {
            NearDf m = s_nf[tid];
#pragma unroll
            for (int w = 1; w < SNW; ++w) m.merge(s_nf[w * TC + tid]);
            if (!m.amb && m.bj >= 0) {
              nnb[tid] = m.bj;
              amb = 0;
            }
          }
        }
        namb[tid] = amb;
      }
      __syncthreads();
      for (int cell = warp; cell < TC; cell += SNW) {
        const int64_t g = c0 + cell;
        if (g >= C || okf[cell] || !namb[cell]) continue;
        const int j = nnb_f64_warp(A.dom, idx, n, A.dom.cell_x[g], A.dom.cell_y[g]);
        if (lane == 0) nnb[cell] = j;
      }
    }
    __syncthreads();
  };

  if (failed) {
    if (tid < TC) {
      okf[tid] = 0;
      cvar[tid] = 0.0;
    }
    if (tid == 0) any_bad = 1;
    nearest();
    for (int e = tid; e < nsteps * TC; e += STC * SNW) emit(e % TC, e / TC, 0.0);
    return;
  }

  double cx = 0.0, cy = 0.0;
  float4 cp[NC];
  __shared__ int wild;  // a cell too far for FP32's squares, or without a place
  __shared__ RhsDf kd;
  __shared__ RhsOne ko;
  // the variogram with its reciprocal ranges (FP64 right-hand sides)
  __shared__ VgPre vgp64;
  if constexpr (sizeof(T) == 8) {
    cx = A.dom.cell_x[gc[0]];
    cy = A.dom.cell_y[gc[0]];
    if (tid == 0) vgp64.init(vg);
  } else {
#pragma unroll
    for (int u = 0; u < NC; ++u) cp[u] = reinterpret_cast<const float4*>(A.dom.cell_split)[gc[u]];
    if (tid == 0) {
      kd.init(vg, sh, A.dom.min_vg_val);
      if (kd.exact && kd.single >= 0) ko.init(kd, vg, sk, sh, A.dom.min_vg_val);
    }
    for (int e = tid; e < 256; e += STC * SNW) s_tab[e] = kExp2.v[e];
    bool w = false;
#pragma unroll
    for (int u = 0; u < NC; ++u) w = w || !(fabsf(cp[u].x) + fabsf(cp[u].z) < kFar);
    w = __syncthreads_or(w) != 0;
    if (tid == 0) {
      wild = w;
      if (w) kd.exact = 0;  // (every entry in FP64)
    }
  }
  const spi_vg_t* vgp = A.sys.vg + s;
  const float4* sp4 = reinterpret_cast<const float4*>(A.dom.stn_split);

  for (int v0 = 0; v0 < nvec; v0 += SSV) {
    const int nv = min(SSV, nvec - v0);
    __syncthreads();
    if (tid < SSV) {
      const int v = v0 + tid;
      const double* p64 = nullptr;
      const float *ph = nullptr, *pl = nullptr;
      if (tid < nv) {
        int64_t off;
        if (v < ndual) {
          off = soff * GA + (int64_t)v * n;
          p64 = A.ws.g_cols + off;
          if (A.ws.g_hi) ph = A.ws.g_hi + off, pl = A.ws.g_lo + off;
        } else {
          off = A.sys.val_off[A.sys.steps[st0 + (v - ndual)]];
          p64 = A.ws.w_hat + off;
          if (A.ws.w_hi) ph = A.ws.w_hi + off, pl = A.ws.w_lo + off;
        }
      }
      vp64[tid] = p64;
      vph[tid] = ph;
      vpl[tid] = pl;
    }
    __syncthreads();
    // (OK / EDK on the Cholesky path pass the sum check on every cell:
    // their sum(lambda) is 1 up to rounding whatever the right-hand side)
    const bool track = sizeof(T) == 4 && fuse_nnb && v0 == 0 && sk;
    NearDf nf[NC];
#pragma unroll
    for (int u = 0; u < NC; ++u) nf[u].init();
    double unit = 1.0;  // of the sums
    if constexpr (sizeof(T) == 8) {
      double acc[SSV];
#pragma unroll
      for (int v = 0; v < SSV; ++v) acc[v] = 0.0;
      for (int j = warp; j < n; j += SNW) {
        const int st = idx[j];
        const double g = vgp64.fill_d2(
            dist2_f64(cx, cy, A.dom.stn_x[st], A.dom.stn_y[st]), sk, A.dom.min_vg_val);
        const double c = (sk || prim) ? g : __dsub_rn(sh, g);
#pragma unroll
        for (int v = 0; v < SSV; ++v)
          if (v < nv) acc[v] = fma(c, vp64[v][j], acc[v]);
      }
#pragma unroll
      for (int v = 0; v < SSV; ++v) red[warp][v][lane] = acc[v];
    } else {
      // double-float entries against hi/lo vectors (stream_chunk)
      float ph[SSV][NC], pl[SSV][NC];
      // the single structure's model, uniform over the CTA; its sums are in
      // units of its sill
      const int scode = (kd.exact && kd.single >= 0 && ko.sill > 0.0) ? kd.code[kd.single] : -1;
      if (scode >= 0) unit = ko.sill;
      const int np = min(max(plain_duals - v0, 0), nv);
#pragma unroll
      for (int v = 0; v < SSV; ++v)
#pragma unroll
        for (int u = 0; u < NC; ++u) {
          ph[v][u] = pl[v][u] = 0.f;
          red[warp][v][u * STC + lane] = 0.0;  // (this thread's alone)
        }
      // stations in chunks staged in shared memory: split coordinates and
      // the vectors' hi/lo pairs, read by every warp at a shared index
      int cnt = 0;
      for (int j0 = 0; j0 < n; j0 += SCH) {
        const int nj = min(SCH, n - j0);
        __syncthreads();
        for (int e = tid; e < nj; e += STC * SNW) {
          // (a gauge beyond kFar is that far from every cell but the wild ones)
          float4 sp = sp4[idx[j0 + e]];
          sp.x = fminf(fmaxf(sp.x, -kFar), kFar);
          sp.z = fminf(fmaxf(sp.z, -kFar), kFar);
          s_sp[e] = sp;
#pragma unroll
          for (int v = 0; v < SSV; ++v)
            if (v < nv) s_w[e][v] = make_float2(vph[v][j0 + e], vpl[v][j0 + e]);
        }
        __syncthreads();
        const int32_t* idxc = idx + j0;
        // compile-time choices: the model, the nearest-station tracking
        // (kernels that never need it carry none of its state through the
        // loop), the vectors of the usual passes
        auto chunk = [&](auto skt, auto trk, auto npt, auto nvt) {
          constexpr bool SK = decltype(skt)::value, TR = decltype(trk)::value;
          constexpr int NP = decltype(npt)::value, NV = decltype(nvt)::value;
#define SPI_STREAM_CHUNK(CODE)                                                                 \
  stream_chunk<CODE, SK, TR, NP, NV>(A, vgp, kd, ko, s_tab, sh, cp, gc, idxc, s_sp, s_w, nj, \
                                     warp, np, nv, ph, pl, nf, j0, esp)
          switch (scode) {
            case SPI_VG_EXP: SPI_STREAM_CHUNK(SPI_VG_EXP); break;
            case SPI_VG_GAU: SPI_STREAM_CHUNK(SPI_VG_GAU); break;
            case SPI_VG_SPH: SPI_STREAM_CHUNK(SPI_VG_SPH); break;
            case SPI_VG_LIN: SPI_STREAM_CHUNK(SPI_VG_LIN); break;
            default: SPI_STREAM_CHUNK(-1);
          }
#undef SPI_STREAM_CHUNK
        };
        using Yes = std::true_type;
        using No = std::false_type;
#define SPI_N(i) std::integral_constant<int, i>{}
        const int form = scode < 0 ? 0 : np * 8 + nv;
        if (track) {
          if (form == 3) chunk(Yes{}, Yes{}, SPI_N(0), SPI_N(3));
          else chunk(Yes{}, Yes{}, SPI_N(-1), SPI_N(-1));
        } else if (sk) {
          if (form == 3) chunk(Yes{}, No{}, SPI_N(0), SPI_N(3));
          else chunk(Yes{}, No{}, SPI_N(-1), SPI_N(-1));
        } else {
          switch (form) {
            case 1: chunk(No{}, No{}, SPI_N(0), SPI_N(1)); break;
            case 2: chunk(No{}, No{}, SPI_N(0), SPI_N(2)); break;
            case 4: chunk(No{}, No{}, SPI_N(0), SPI_N(4)); break;
            case 10: chunk(No{}, No{}, SPI_N(1), SPI_N(2)); break;
            case 12: chunk(No{}, No{}, SPI_N(1), SPI_N(4)); break;
            case 20: chunk(No{}, No{}, SPI_N(2), SPI_N(4)); break;
            case 19: chunk(No{}, No{}, SPI_N(2), SPI_N(3)); break;
            case 28: chunk(No{}, No{}, SPI_N(3), SPI_N(4)); break;
            default: chunk(No{}, No{}, SPI_N(-1), SPI_N(-1));
          }
        }
#undef SPI_N
        cnt += SCH / SNW;
        if (cnt >= 256 || j0 + SCH >= n) {
          cnt = 0;
#pragma unroll
          for (int v = 0; v < SSV; ++v)
#pragma unroll
            for (int u = 0; u < NC; ++u) {
              red[warp][v][u * STC + lane] += (double)ph[v][u] + (double)pl[v][u];
              ph[v][u] = pl[v][u] = 0.f;
            }
        }
      }
    }
    __syncthreads();
    for (int e = tid; e < nv * TC; e += STC * SNW) {
      const int v = e / TC, cell = e % TC;
      double t = 0.0;
#pragma unroll
      for (int w = 0; w < SNW; ++w) t += red[w][v][cell];
      vres[v][cell] = t * unit;
    }
    __syncthreads();
    if (track) {
      // red is free again
#pragma unroll
      for (int u = 0; u < NC; ++u) s_nf[warp * TC + u * STC + lane] = nf[u];
      nf_ready = !wild;
    }
    for (int e = tid; e < nv * TC; e += STC * SNW)
      if (v0 + e / TC < ndual) qsh[v0 + e / TC][e % TC] = vres[e / TC][e % TC];
    __syncthreads();
    if (v0 < ndual && v0 + nv >= ndual) {
      // the sum check of every cell, once its dual columns are complete
      if (tid == 0) any_bad = any_chk = 0;
      __syncthreads();
      if (tid < TC) {
        const int cell = tid;
        const int64_t g = c0 + cell;
        double q[GA], f[GA], nu[GA];
        for (int k = 0; k < GA; ++k) q[k] = k < ndual ? qsh[k][cell] : 0.0;
        f[0] = 1.0;
        for (int k = 1; k < GA; ++k)
          f[k] = (k < a && g < C && !sk) ? A.dom.cell_drift[(int64_t)(k - 1) * C + g] : 0.0;
        double sl;
        if (prim) {
          sl = q[0];
          if (!sk)
            for (int k = 0; k < a; ++k) sl += f[k] * A.ws.g_colsum[(int64_t)s * GA + k];
        } else if (sk) {
          sl = q[0];
        } else {
          const double* Si = A.ws.s_inv + (int64_t)s * GA * GA;
          for (int k = 0; k < a; ++k) {
            double t = 0.0;
            for (int l = 0; l < a; ++l) t += Si[k * GA + l] * (q[l] - f[l]);
            nu[k] = t;
          }
          sl = q[0];
          for (int k = 0; k < a; ++k) sl -= A.ws.g_colsum[(int64_t)s * GA + k] * nu[k];
          if (var_out && g < C)
            cvar[cell] = sh * sl - A.ws.cell_yy[(int64_t)s * C + g] + nu[0] * q[0] - 2.0 * nu[0];
        }
        int ok = isclose_one(sl) ? 1 : 0;
        // SK's FP32 sum(lambda) within its rounding bound of the check's
        // boundary: decided in FP64 (as k_krige_cells)
        if (sizeof(T) == 4 && sk && g < C &&
            near_isclose_boundary(sl, kSumLambdaRelErrDf * q[1])) {
          ok = 2;
          atomicOr(&any_chk, 1);
        }
        okf[cell] = ok;
        if (!ok && g < C) atomicOr(&any_bad, 1);
      }
      __syncthreads();
      if (any_chk)
        for (int cell = warp; cell < TC; cell += SNW) {
          if (okf[cell] != 2) continue;
          const int64_t g = c0 + cell;
          const double sl = sk_sum_lambda_f64(A.dom, vg, idx, n, A.ws.g_cols + soff * GA,
                                              A.dom.cell_x[g], A.dom.cell_y[g]);
          if (lane == 0) {
            const int ok = isclose_one(sl) ? 1 : 0;
            okf[cell] = ok;
            if (!ok) atomicOr(&any_bad, 1);
          }
        }
      nearest();
    }
    for (int e = tid; e < nv * TC; e += STC * SNW) {
      const int v = v0 + e / TC, cell = e % TC;
      if (v >= ndual) emit(cell, v - ndual, vres[e / TC][cell]);
    }
  }
}

int launch_cells_stream(const CellsArgs& A, int precision, cudaStream_t st) {
  const int tc = precision == 0 ? STC : STC * SC4;
  const int64_t tiles = (A.dom.n_cells + tc - 1) / tc;
  if (tiles > 0x7fffffff) return SPI_ERR_TOO_LARGE;
  dim3 grid((unsigned)tiles, (unsigned)A.sys.n_sys);
  const bool f64 = A.out.out_f64 != 0;
  if (precision == 0) {
    if (f64) k_krige_cells_stream<double, double><<<grid, STC * SNW, 0, st>>>(A);
    else k_krige_cells_stream<double, float><<<grid, STC * SNW, 0, st>>>(A);
  } else {
    if (f64) k_krige_cells_stream<float, double><<<grid, STC * SNW, 0, st>>>(A);
    else k_krige_cells_stream<float, float><<<grid, STC * SNW, 0, st>>>(A);
  }
  SPI_LAUNCH_CHECK();
  return SPI_OK;
}

}  // namespace spi
