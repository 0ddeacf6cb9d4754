// Covariance entries in 64-bit fixed point.
//
// GB300 issues an FP64 operation at 1/64 of the rate of an integer or FP32
// one, and an entry in FP64 (two differences, a square root, an exponential)
// is about 45 of them. Here an entry is about 200 integer operations, the
// 32 x 32 -> 64 bit products among them at half rate: the coordinates as
// 62-bit integers on a common grid, the distance's square and root by
// normalised 64-bit products, the model in fixed point. The result is the
// correlation-like c / (the structures' sills) as an integer of FX_BITS = 62 bits with an
// error of about 2^-56 of those sills (rms 2^-58 for one structure), where an
// FP64 evaluation is off by 2^-54 (rms). That holds on a grid that is fine
// enough for the structures' ranges (fx_resolves); others keep FP64.
//
// The functions are host and device code, so that their error can be
// measured against wider arithmetic on the CPU.
#pragma once
#include <cmath>
#include <cstdint>

#include <cuda_runtime.h>

#include "spinterps_gb300.h"

namespace spi {

constexpr int FX_BITS = 62;                    // an entry of the structures' sills is 2^62
constexpr int FX_GRID = 61;                    // coordinates without an origin: |X| <= 2^61

#define FX_HD __host__ __device__ __forceinline__

FX_HD uint64_t fx_mulhi(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}
// The high word of a product to within 2 units: the product of the low
// halves left out (7 instructions instead of 12), 1 added for its mean and
// the dropped fractions'.
FX_HD uint64_t fx_mulh(uint64_t a, uint64_t b) {
  const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a;
  const uint32_t bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
  return (uint64_t)ah * bh + (uint32_t)(((uint64_t)ah * bl) >> 32) +
         (uint32_t)(((uint64_t)al * bh) >> 32) + 1;
}
// The same of a square.
FX_HD uint64_t fx_sqrh(uint64_t a) {
  const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a;
  return (uint64_t)ah * ah + (((uint64_t)ah * al) >> 31);
}
FX_HD int fx_clz(uint64_t a) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)a);
#else
  return a ? __builtin_clzll(a) : 64;
#endif
}
FX_HD float fx_rsqrt(float x) {
#ifdef __CUDA_ARCH__
  return rsqrtf(x);
#else
  return 1.0f / sqrtf(x);
#endif
}

FX_HD float fx_rcpf(float x) {
#ifdef __CUDA_ARCH__
  return __fdividef(1.0f, x);
#else
  return 1.0f / x;
#endif
}

// The common grid of a domain: X = (x - ox) 2^q.
struct FxGrid {
  double ox, oy;
  int q;
  int exact;  // it holds every point exactly
};

// It, and whether the points have one (finite, not past FP64's middle range).
struct FxScene {
  FxGrid g;
  int ok;
};

// The place of x's last bit, x = odd 2^place: a grid of 2^-q holds x exactly
// where it is -q or more.
FX_HD int fx_place(double x) {
#ifdef __CUDA_ARCH__
  const int64_t b = __double_as_longlong(x);
#else
  int64_t b;
  __builtin_memcpy(&b, &x, 8);
#endif
  const int e = (int)((b >> 52) & 0x7ff);
  const int64_t m = (b & 0xfffffffffffffll) | (e ? 1ll << 52 : 0);
  if (m == 0) return 4096;
  return (e ? e : 1) - 1075 + 63 - fx_clz((uint64_t)(m & -m));
}

// The grid of points between (x0, y0) and (x1, y1): its origin in
// their middle, so that |X| <= 2^62 (a difference stays under 2^63) with a step
// of 2^-63 to 2^-62 of the larger side. False where it has none. place: the
// finest place of the points' coordinates (fx_place), or less.
FX_HD bool fx_grid(double x0, double x1, double y0, double y1, int place, FxGrid& g) {
  const double dx = x1 - x0, dy = y1 - y0;
  double ext = fmax(dx, dy);
  g.ox = x0 + 0.5 * dx;
  g.oy = y0 + 0.5 * dy;
  const bool ok = dx >= 0.0 && dy >= 0.0 && ext < 1e200 && x0 > -1e250 && y0 > -1e250;
  if (!(ext > 1e-200)) ext = 1e-200;
  int e = 0;
  frexp(ext, &e);
  g.q = FX_GRID + 2 - e;
  const int po = fx_place(g.ox) < fx_place(g.oy) ? fx_place(g.ox) : fx_place(g.oy);
  g.exact = (place < po ? place : po) >= -g.q;
  return ok;
}

// Whether the grid is fine enough for a variogram. It is where it holds the
// points exactly (coordinates of some size of their own, as projected ones:
// their last place is that of 2^-52 of it). Else its rounding moves a
// distance by 0.41 steps (rms: four coordinates, a third of them each way), so
// an entry by 0.41 steps times the structures' slopes at their steepest, if no
// coordinate is exact on it (in practice most are). The 2^-54 of the
// sills that an FP64 evaluation is off by (rms) bounds that; a structure of
// little sill counts little. Measured against 113-bit arithmetic (Exp, pairs
// within the range, coordinates near 0; rms in units of 2^-54 of the sill, FP64
// 1.05): extent / range 128 0.03, 200 (the limit lies between 170 and 340 by
// the extent's binary place) 0.05, 500 0.20, 2100 1.7, 8500 7.
FX_HD bool fx_resolves(const spi_vg_t& vg, const FxGrid& g) {
  if (g.exact) return true;
  double tot = 0.0, slope = 0.0;
  for (int c = 0; c < vg.n_comp; ++c) {
    if (vg.code[c] == SPI_VG_NUG) continue;
    const double k = vg.code[c] == SPI_VG_EXP ? 3.0 : (vg.code[c] == SPI_VG_LIN ? 1.0 : 1.5);
    tot += vg.sill[c];
    slope += k * vg.sill[c] / vg.range[c];
  }
  return slope <= tot * ldexp(1.0, g.q - 53);
}

// x - o on the grid, the difference's rounding error included.
FX_HD int64_t fx_coord(double x, double o, int q) {
  const double d = x - o;
  const double b = d - x;
  const double e = (x - (d - b)) - (o + b);
  return llrint(ldexp(d, q)) + llrint(ldexp(e, q));
}

// x on the grid without an origin, by integer shifts: X = x 2^q, for
// |x| < 2^(FX_GRID - q); places finer than the grid are cut off.
FX_HD int64_t fx_coord0(double x, int q) {
#ifdef __CUDA_ARCH__
  const int64_t b = __double_as_longlong(x);
#else
  int64_t b;
  __builtin_memcpy(&b, &x, 8);
#endif
  const int e = (int)((b >> 52) & 0x7ff);
  const int64_t m = (b & 0xfffffffffffffll) | (e ? 1ll << 52 : 0);
  const int sh = (e ? e : 1) - 1075 + q;  // x = m 2^(e - 1075)
  const int64_t v = sh >= 0 ? m << (sh < 63 ? sh : 63) : m >> (-sh < 63 ? -sh : 63);
  return b < 0 ? -v : v;
}

// A positive double as a 64-bit mantissa and an exponent: v = m 2^e, m with
// its top bit set.
FX_HD void fx_norm(double v, uint64_t& m, int& e) {
  int x;
  const double f = frexp(v, &x);             // [0.5, 1)
  m = (uint64_t)ldexp(f, 53) << 11;
  e = x - 64;
}

// What one structure needs: its weight in the structures' sills (Q64) and the
// scaled reciprocal range k 2^-q (or k 2^-2q) as a normalised mantissa.
struct FxComp {
  uint64_t w, km;
  int code, sh;  // sh: see fx_rho
};

struct FxVg {
  FxComp c[SPI_MAX_VG_COMP];
  int n;          // structures (nuggets add nothing to a covariance)
  int ok;         // every structure has a form here
  int sk;
  int64_t cut;    // min_vg_val's boundary, in units; < 0: no cut
  int64_t over;   // what an entry past the cut becomes
  double sill;    // the structures' total sill: an entry's unit is sill 2^-FX_BITS
};

// x / y of two positive doubles as Q64 (x <= y; the ratio 1 saturates).
FX_HD uint64_t fx_ratio(double x, double y) {
  const double r = x / y;
  if (r >= 1.0) return ~0ull;
  const double rem = fma(-r, y, x) / y;      // the quotient's rounding error
  const uint64_t hi = (uint64_t)ldexp(r, 64);
  return hi + (uint64_t)(int64_t)llrint(ldexp(rem, 64));
}

// k / d as a normalised 64-bit mantissa and exponent (k, d > 0).
FX_HD void fx_recip(double k, double k_lo, double d, uint64_t& m, int& e) {
  const double r = k / d;
  const double rem = (fma(-r, d, k) + k_lo) / d;
  fx_norm(r, m, e);
  // the mantissa's unit is 2^e; add the remainder in that unit
  const int64_t a = llrint(ldexp(rem, -e));
  const uint64_t s = m + (uint64_t)a;
  if (a < 0 && s > m) m = 0, --e;  // not reached: m >= 2^63 and |a| < 2^11
  else if (a >= 0 && s < m) m = ~0ull;
  else m = s;
}

FX_HD void fx_init(FxVg& f, const spi_vg_t& vg, int sk, double min_vg_val, int q) {
  f.n = 0;
  f.ok = 1;
  f.sk = sk;
  double tot = 0.0, all = 0.0;
  for (int c = 0; c < vg.n_comp; ++c) {
    all += vg.sill[c];
    if (vg.code[c] != SPI_VG_NUG) tot += vg.sill[c];
  }
  f.sill = tot;
  f.cut = -1;
  f.over = 0;
  if (!(tot > 0.0) || !(all < 1e300)) f.ok = 0;
  // 3 / ln 2 as two doubles
  const double k3 = 4.328085122666891, k3l = -3.830233886272695e-16;
  for (int c = 0; c < vg.n_comp; ++c) {
    const int code = vg.code[c];
    if (code == SPI_VG_NUG) continue;
    FxComp& o = f.c[f.n];
    o.code = code;
    const double r = vg.range[c];
    if (!(vg.sill[c] >= 0.0) || !(r > 0.0) || !(r < 1e150)) f.ok = 0;
    if (!f.ok) return;
    o.w = fx_ratio(vg.sill[c], tot);
    int e = 0;
    // the product of the normalised distance (or its square) with km, shifted
    // right by L + sh (2 L + sh), is t in Q56 (Exp, Gau) or Q62 (Sph, Lin)
    if (code == SPI_VG_EXP) {
      fx_recip(k3, k3l, r, o.km, e);
      o.sh = -(121 + e - q);
    } else if (code == SPI_VG_GAU) {
      // r^2 as a double-double: its rounding error joins the numerator's
      const double r2 = r * r, r2l = fma(r, r, -r2);
      fx_recip(k3, k3l - k3 * (r2l / r2), r2, o.km, e);
      o.sh = -(186 + e - 2 * q);
    } else if (code == SPI_VG_SPH || code == SPI_VG_LIN) {
      fx_recip(1.0, 0.0, r, o.km, e);
      o.sh = -(127 + e - q);
    } else {
      f.ok = 0;
      return;
    }
    ++f.n;
  }
  if (min_vg_val > 0.0) {
    // SK: an entry <= min_vg_val becomes 0. OK / EDK: gamma <= min_vg_val,
    // an entry >= all - min_vg_val (all the sills, nuggets included),
    // becomes all; nuggets above the cut keep every entry under it
    const double x = (sk ? min_vg_val : all - min_vg_val) / tot, o = sk ? 0.0 : all / tot;
    if (sk ? x >= 1.0 : (x <= 0.0 || (x <= 1.0 && o > 1.25))) {
      f.ok = 0;  // (everything cut, or an entry beyond the digits' range)
    } else if (x <= 1.0) {
      f.cut = llrint(ldexp(x, FX_BITS));
      f.over = llrint(ldexp(o, FX_BITS));
    }
  }
}

// 2^-(2^-k), k = 1..8, as Q64: the factors of the table 2^(-j / 256).
FX_HD uint64_t fx_exp2_factor(int k) {
  const uint64_t t[8] = {0xb504f333f9de6484ull, 0xd744fccad69d6af4ull, 0xeac0c6e7dd24392full,
                         0xf5257d152486cc2cull, 0xfa83b2db722a033aull, 0xfd3e0c0cf486c175ull,
                         0xfe9e115c7b8f884cull, 0xff4ecb59511ec8a5ull};
  return t[k - 1];
}
// Table entry 2^(-j / 256) as Q63.
FX_HD uint64_t fx_exp2_entry(int j) {
  uint64_t v = 1ull << 63;
  for (int k = 1; k <= 8; ++k)
    if (j & (256 >> k)) v = fx_mulhi(v, fx_exp2_factor(k));
  return v;
}

// 2^-t for t in Q56 as an integer of FX_BITS bits: 2^-(integer part) by the
// shift, 2^-(j / 256) from the table, the rest x 2^-8 (x < 1) by its Taylor
// polynomial of degree 5 (the next term is 2^-60), each coefficient in the
// precision that its place in the sum needs.
FX_HD int64_t fx_exp2(uint64_t t, const uint64_t* tab) {
  const int m = (int)(t >> 56);
  const uint64_t T = tab[(t >> 48) & 255];
  const uint64_t x = t << 16;  // Q64
  const uint32_t xh = (uint32_t)(x >> 32);
  // c5 2^30, c4 2^38, c3 2^36 (Q62, Q62, Q52 of c_k 2^-8(k-1)); c2 2^56 and
  // c1 2^64 (Q64), c_k = ln2^k / k!
  const uint32_t v4 = 2643811198u - (uint32_t)(((uint64_t)xh * 1431680u) >> 32);
  const uint32_t v3 = 3814213304u - ((uint32_t)(((uint64_t)xh * v4) >> 32) >> 10);
  const uint64_t v2 = 17310144115608349ull - (((uint64_t)xh * v3) >> 20);
  const uint64_t v1 = 12786308645202655660ull - fx_mulh(x, v2);
  const uint64_t d = fx_mulh(x, v1);               // 2^8 (1 - 2^-(x 2^-8)), Q64
  const uint64_t r = T - (fx_mulh(T, d) >> 8);     // Q63
  const int sh = 63 - FX_BITS + m;
  return sh > 63 ? 0 : (int64_t)((r + (1ull << (sh - 1))) >> sh);
}

// sqrt(S) 2^32 of S in [2^60, 2^63): a 31-bit root from FP32 (a relative
// 2^-21), then two corrections by the exact remainder (2^-46, 2^-62).
FX_HD uint64_t fx_sqrt(uint64_t S) {
  const float f = (float)(uint32_t)(S >> 32);       // S 2^-32
  const float y = fx_rsqrt(f);                      // 2^16 / sqrt(S)
  const uint32_t h0 = (uint32_t)(f * y * 65536.0f);
  // E = S - h0^2, |E| < 2^43; E / (2 h0) with 16 fraction bits
  const int64_t E = (int64_t)(S - (uint64_t)h0 * h0);
  const int32_t i1 = (int32_t)rintf((float)(int32_t)(E >> 16) * y * 32768.0f);
  const uint64_t H = ((uint64_t)h0 << 32) + (uint64_t)((int64_t)i1 << 16);
  // (S 2^64 - H^2) 2^-32 modulo 2^64 (its size is under 2^51)
  const int64_t E1 = (int64_t)(((uint64_t)E << 32) - ((uint64_t)((int64_t)i1 * (int64_t)h0) << 17) -
                               (uint64_t)((int64_t)i1 * i1));
  // its correction E1 2^32 / (2 H)
  const int32_t i2 = (int32_t)rintf((float)(int32_t)(E1 >> 24) * y * 128.0f);
  return H + (uint64_t)(int64_t)i2;
}

// 2^126 / M in Q62 of a normalised M (top bit set): FP32's reciprocal, then
// two Newton steps (relative 2^-44, 2^-60).
FX_HD uint64_t fx_rcp(uint64_t M) {
  const float y = fx_rcpf((float)(uint32_t)(M >> 32));
  uint64_t R = (uint64_t)(uint32_t)(y * 4611686018427387904.0f) << 32;
  int64_t E = (int64_t)((1ull << 62) - fx_mulh(M, R));  // (1 - m r) 2^62
  R += (uint64_t)(((int64_t)(R >> 32) * (int32_t)(E >> 16)) >> 14);
  E = (int64_t)((1ull << 62) - fx_mulh(M, R));
  return R + (uint64_t)(((int64_t)(R >> 32) * (int32_t)E) >> 30);
}

// A cell-station distance on the grid: S = h^2 2^(2 L - 66) in [2^60, 2^63),
// 0 when the points coincide.
struct FxDist {
  uint64_t S;
  int L;
};
FX_HD FxDist fx_dist(int64_t cx, int64_t cy, int64_t sx, int64_t sy) {
  const int64_t dx = cx - sx, dy = cy - sy;
  uint64_t ax = (uint64_t)(dx < 0 ? -dx : dx), ay = (uint64_t)(dy < 0 ? -dy : dy);
  const int L = fx_clz((ax | ay) | 1);
  ax <<= L;
  ay <<= L;
  return {(fx_sqrh(ax) >> 2) + (fx_sqrh(ay) >> 2), L};
}

// A correlation times its structure's weight.
FX_HD int64_t fx_weighed(int64_t v, uint64_t w) {
  return w == ~0ull ? v : (int64_t)(fx_mulh((uint64_t)v << 1, w) >> 1);
}

// One structure's correlation, its weight included; H: fx_sqrt(S) =
// h 2^(L - 1) (not read by Gau). No branches on data: a warp's lanes keep
// together.
FX_HD int64_t fx_rho(int code, const FxComp& k, FxDist d, uint64_t H, const uint64_t* tab) {
  int64_t v;
  if (code == SPI_VG_GAU) {
    const int z = fx_clz(d.S | 1);
    const uint64_t T = fx_mulh(d.S << z, k.km);
    const int sh = 2 * d.L + z + k.sh;
    v = fx_exp2(T >> (sh < 0 ? 0 : (sh > 63 ? 63 : sh)), tab);
    v = sh < 0 ? 0 : v;
  } else {
    const uint64_t T = fx_mulh(H, k.km);
    const int sh = d.L + k.sh;
    // (a negative shift: Exp past 2^-64; h / r >= 1, as T >= 2^61)
    const uint64_t t0 = T >> (sh < 0 ? 0 : (sh > 63 ? 63 : sh));
    if (code == SPI_VG_EXP) {
      v = fx_exp2(t0, tab);
      v = sh < 0 ? 0 : v;
    } else {
      // h / r in Q62
      const bool out = sh < 0 || t0 >= (1ull << 62);
      if (code == SPI_VG_LIN) {
        v = (int64_t)((1ull << 62) - t0);
      } else {
        // 1 - t (3 - t^2) / 2
        const uint64_t t = t0 << 1;                             // Q63
        const uint64_t t2 = fx_mulh(t, t);                     // Q62
        const uint64_t b = fx_mulh(t, (3ull << 62) - t2);      // Q61
        v = ((int64_t)1 << FX_BITS) - (int64_t)b;
      }
      v = out ? 0 : v;
    }
  }
  v = d.S == 0 ? (int64_t)1 << FX_BITS : v;
  return fx_weighed(v, k.w);
}

// N entries of one cell, before the min_vg_val cut. CODE: the model of a
// variogram with one structure, known at compile time (its instructions
// then interleave over the entries), or -1.
template <int CODE, int N>
FX_HD void fx_entries(const FxVg& f, const FxDist (&d)[N], const uint64_t* tab, int64_t (&v)[N]) {
  uint64_t H[N];
  if (CODE < 0 || CODE != SPI_VG_GAU)
    for (int e = 0; e < N; ++e) H[e] = fx_sqrt(d[e].S);
  if (CODE >= 0) {
    const FxComp k = f.c[0];
    for (int e = 0; e < N; ++e) v[e] = fx_rho(CODE, k, d[e], H[e], tab);
  } else {
    for (int e = 0; e < N; ++e) v[e] = 0;
    for (int c = 0; c < f.n; ++c) {
      const FxComp k = f.c[c];
      for (int e = 0; e < N; ++e) v[e] += fx_rho(k.code, k, d[e], H[e], tab);
    }
  }
}

// One entry (the same arithmetic).
FX_HD int64_t fx_entry(const FxVg& f, int64_t cx, int64_t cy, int64_t sx, int64_t sy,
                       const uint64_t* tab) {
  const FxDist d[1] = {fx_dist(cx, cy, sx, sy)};
  int64_t v[1];
  fx_entries<-1, 1>(f, d, tab, v);
  return v[0];
}

// An integer v < 2^63 as a double times 2^-FX_BITS, by its bits (no FP64
// operation), rounded.
FX_HD double fx_double(uint64_t v) {
  const int c = fx_clz(v | 1);
  const uint64_t m = ((v << c) >> 11) + (((v << c) >> 10) & 1);
  // (a carry into the exponent comes out right)
  const uint64_t b = v ? ((uint64_t)(1022 + 63 - FX_BITS - c) << 52) + m : 0;
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double w;
  __builtin_memcpy(&w, &b, 8);
  return w;
#endif
}

// A squared distance as a monotone key: the exponent above 55 bits of the
// normalised square (its top bit set). 0: the points coincide.
constexpr int FX_KEY = 511;
FX_HD uint64_t fx_key(FxDist d) {
  const int z = fx_clz(d.S | 1);
  return d.S ? ((uint64_t)(FX_KEY - 2 * d.L - z) << 55) + ((d.S << z) >> 9) : 0ull;
}

// The same form of a squared distance d2 > 0 given in FP64 (normal), on a grid
// of 2^-q: what lies too close for the grid. Distances under 2^-191 steps
// count as that.
FX_HD FxDist fx_dist_f64(double d2, int q) {
#ifdef __CUDA_ARCH__
  const int64_t b = __double_as_longlong(d2);
#else
  int64_t b;
  __builtin_memcpy(&b, &d2, 8);
#endif
  const int e = (int)(b >> 52) - 1022;  // d2 = f 2^e, f in [1/2, 1)
  const int t = 128 - e - 2 * q, L = t >> 1;
  const uint64_t m = (uint64_t)((b & 0xfffffffffffffll) | (1ll << 52));
  if (L > 254) return {1ull << 60, 254};
  return {m << (9 - (t & 1)), L};
}

// The inverse-square weight (h_ref / h)^2 <= 1 as a double, by its bits (no
// FP64 operation); ref: the key of the smallest distance. Relative error
// 2^-53 (the rounding) and a few 2^-59. d.S != 0.
FX_HD double fx_weight2(FxDist d, uint64_t ref) {
  const int z = fx_clz(d.S | 1);
  const uint64_t q = fx_mulh((ref & ((1ull << 55) - 1)) << 9, fx_rcp(d.S << z));  // Q62
  const int c = fx_clz(q);
  // the top 53 bits, rounded (a carry into the exponent comes out right)
  const uint64_t m = ((q << c) >> 11) + (((q << c) >> 10) & 1);
  const int e = 1024 - c - ((FX_KEY - 2 * d.L - z) - (int)(ref >> 55));
  const uint64_t b = ((uint64_t)(e - 1) << 52) + m;
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double w;
  __builtin_memcpy(&w, &b, 8);
  return w;
#endif
}

}  // namespace spi
