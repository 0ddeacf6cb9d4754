// Neighbour selection of every destination cell among a set of reference
// stations: SpInterpNeighborGrouping's 'nrst' and 'pie' methods
// (interp/grps.py:147-247 with cyth/interpmthds.pyx:811-890), one thread per
// destination, results as each destination's sorted station indices.
//
// nrst: the n_nebs nearest (FP64 distances, the correctly rounded root as
// numpy's ** 0.5), ordered by (distance, index) (k_neb_nrst).
// pie: every station's angle from the destination by the reference's rules
// (atan(dy / dx), pushed into [0, 2 pi) for dx < 0 or dy < 0 -- dx == 0
// gives 0, and dx < 0 with dy == 0 stays 0), its pie
// int(angle * n_pies / 2 pi), its rank by distance within its pie; the
// stations ordered by (rank, distance) -- the nearest of every pie first --
// and the first n_nebs taken (k_neb_pie).
//
// Both kernels decide in FP32 what FP32 can decide and give the rest (a tie
// within its rounding, a direction at a pie's edge) to the FP64 rule: FP64
// operations issue at 1/64 of FP32's rate here.
//
// Ties: the reference orders equal distances with numpy's (unstable)
// argsort; here they order by index. A pie index that rounds up to n_pies
// (an angle within an ulp of 2 pi, where the reference writes past its
// count array) is taken as the last pie.
#include "spi_common.cuh"

namespace spi {

constexpr int NEB_MAX = 64;
constexpr int NEB_PIE_SLOTS = 512;   // n_pies * n_nebs

__device__ __forceinline__ bool neb_less(double da, int ia, double db, int ib) {
  return da < db || (da == db && ia < ib);
}

// insert (d, i) into the ascending list (ld, li) of length *len (cap k)
__device__ __forceinline__ void neb_insert(double* ld, int* li, int* len, int k, double d, int i) {
  int n = *len;
  if (n == k && !neb_less(d, i, ld[n - 1], li[n - 1])) return;
  int p = (n == k) ? n - 1 : n;
  while (p > 0 && neb_less(d, i, ld[p - 1], li[p - 1])) {
    ld[p] = ld[p - 1];
    li[p] = li[p - 1];
    --p;
  }
  ld[p] = d;
  li[p] = i;
  if (n < k) *len = n + 1;
}

__device__ __forceinline__ void sort_ints(int* a, int n) {
  for (int i = 1; i < n; ++i) {
    int v = a[i], p = i;
    while (p > 0 && a[p - 1] > v) {
      a[p] = a[p - 1];
      --p;
    }
    a[p] = v;
  }
}

// Stations pass through shared memory in tiles as FP32 coordinates relative
// to station 0, with |x| + |y| beside them. The rounding of the FP32
// coordinates and arithmetic moves a distance by at most 2^-23 (|x_s| + |y_s|
// + |x_c| + |y_c|) plus a few 1e-7 of it; NEB_ABS = 2^-20 and NEB_REL = 1e-5
// bound both with room to spare.
constexpr int NEB_T = 128;      // threads per CTA
constexpr int NEB_TILE = 1024;  // stations per shared-memory tile
constexpr float NEB_REL = 1.00001f;
constexpr float NEB_ABS = 0x1p-20f;

struct NebCell {
  double x, y;
  float xc, yc, sc;
};
__device__ __forceinline__ NebCell neb_cell(const double* dx_, const double* dy_, int64_t i,
                                            bool act, double ox, double oy) {
  NebCell c;
  c.x = act ? dx_[i] : ox;
  c.y = act ? dy_[i] : oy;
  c.xc = (float)(c.x - ox);
  c.yc = (float)(c.y - oy);
  c.sc = fabsf(c.xc) + fabsf(c.yc);
  return c;
}
// The bounds hold while nothing overflows, and underflow stays below them.
__device__ __forceinline__ bool neb_in_range(float size) { return size > 1e-15f && size < 1e18f; }
// every thread of the CTA: the tile of stations from t0 on; its size. bad: set
// where a coordinate is not finite.
__device__ __forceinline__ int neb_tile(float4* tile, const double* rx, const double* ry,
                                        int n_ref, int t0, double ox, double oy, bool& bad) {
  const int tn = min(NEB_TILE, n_ref - t0);
  __syncthreads();
  for (int j = threadIdx.x; j < tn; j += NEB_T) {
    const float xs = (float)(rx[t0 + j] - ox), ys = (float)(ry[t0 + j] - oy);
    const float z = fabsf(xs) + fabsf(ys);
    tile[j] = make_float4(xs, ys, z, 0.0f);
    bad = bad || !(z < INFINITY);
  }
  bad = __syncthreads_or(bad) != 0;
  return tn;
}
__device__ __forceinline__ float neb_d2(const NebCell& c, float4 s) {
  const float ex = s.x - c.xc, ey = s.y - c.yc;
  return fmaf(ex, ex, ey * ey);
}

// Station j outside the tile loops: from the tile while that holds them all.
__device__ __forceinline__ float4 neb_stn(const float4* tile, const double* rx, const double* ry,
                                          int n_ref, int j) {
  if (n_ref <= NEB_TILE) return tile[j];
  const float xs = (float)(rx[j] - rx[0]), ys = (float)(ry[j] - ry[0]);
  return make_float4(xs, ys, fabsf(xs) + fabsf(ys), 0.0f);
}

// Candidates of one destination that its warp puts in order together.
constexpr int NEB_CAND = 128;
struct NebCand {
  double d[NEB_CAND];
  int j[NEB_CAND], key[NEB_CAND];
};
// lane src's destination, to every lane
__device__ __forceinline__ NebCell neb_share(const NebCell& c, int src) {
  NebCell o;
  o.x = __shfl_sync(0xffffffffu, c.x, src);
  o.y = __shfl_sync(0xffffffffu, c.y, src);
  o.xc = __shfl_sync(0xffffffffu, c.xc, src);
  o.yc = __shfl_sync(0xffffffffu, c.yc, src);
  o.sc = __shfl_sync(0xffffffffu, c.sc, src);
  return o;
}
// Appends the lanes' hits in lane order; n: their number so far.
__device__ __forceinline__ void neb_append(NebCand& w, bool hit, int j, int key, int& n) {
  const int lane = threadIdx.x % 32;
  const unsigned m = __ballot_sync(0xffffffffu, hit);
  const int at = n + __popc(m & ((1u << lane) - 1));
  if (hit && at < NEB_CAND) {
    w.j[at] = j;
    w.key[at] = key;
  }
  n += __popc(m);
}
// The k candidates (ascending j) of the smallest place, in ascending order.
template <typename F>
__device__ __forceinline__ void neb_take(const NebCand& w, int n, int k, int32_t* o, F place) {
  const int lane = threadIdx.x % 32;
  int cnt = 0;
  for (int e0 = 0; e0 < n; e0 += 32) {
    const int e = e0 + lane;
    const bool sel = e < n && place(e) < k;
    const unsigned m = __ballot_sync(0xffffffffu, sel);
    if (sel) o[cnt + __popc(m & ((1u << lane) - 1))] = w.j[e];
    cnt += __popc(m);
  }
}

// The k nearest by (FP64 distance, index) over every station.
__device__ __noinline__ void neb_nrst_exact(const NebCell& c, const double* rx, const double* ry,
                                            int n_ref, int k, int32_t* out) {
  double ld[NEB_MAX];
  int li[NEB_MAX];
  int len = 0;
  for (int j = 0; j < n_ref; ++j)
    neb_insert(ld, li, &len, k, dist_f64(c.x, c.y, rx[j], ry[j]), j);
  sort_ints(li, len);
  for (int q = 0; q < k; ++q) out[q] = li[q];
}

// nrst: a first scan keeps the K smallest squared FP32 distances sorted in
// registers (K >= k, the surplus slots hold -1, so that the last slot is the
// k-th smallest, T); an insertion is 2 K minima and maxima, without branches
// on data inside. No k-th nearest lies beyond
//   U = sqrt(T) (1 + 1e-5) + 2^-20 (max |x_s| + |y_s| + |x_c| + |y_c|),
// so a station with an FP32 distance above
//   U (1 + 1e-5) + 2^-20 (|x_s| + |y_s| + |x_c| + |y_c|)
// is none of the k. The second scan writes the others out as they come, in
// ascending index; where they are exactly k they are the answer, whatever
// their order, else (a tie within the rounding) the destination's warp puts
// them in order by their FP64 distances, a candidate to a lane; where a
// coordinate is not finite or beyond the bounds' range, every station is, by
// the destination's thread.
//
// Bound by the scans' latency (about 13 warps to an SM at 62 500
// destinations). 16 of 750 stations there: 1.06 ms with FP64 insertion lists
// in local memory, 0.27 with these lists and ties left to a thread, 0.076 now.
// Four threads to a destination take longer (0.33): four lists make more
// insertions than one.
template <int K>
__global__ __launch_bounds__(NEB_T) void k_neb_nrst(const double* __restrict__ dx_,
                                                    const double* __restrict__ dy_,
                                                    int64_t n_dst,
                                                    const double* __restrict__ rx,
                                                    const double* __restrict__ ry, int n_ref,
                                                    int k, int32_t* __restrict__ out) {
  __shared__ float4 tile[NEB_TILE];
  __shared__ NebCand cand[NEB_T / 32];
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const bool act = i < n_dst;
  const double ox = rx[0], oy = ry[0];
  const NebCell c = neb_cell(dx_, dy_, i, act, ox, oy);
  float a[K];
#pragma unroll
  for (int q = 0; q < K; ++q) a[q] = q < K - k ? -1.0f : INFINITY;
  float smax = 0.0f;
  bool bad = false;
  for (int t0 = 0; t0 < n_ref; t0 += NEB_TILE) {
    const int tn = neb_tile(tile, rx, ry, n_ref, t0, ox, oy, bad);
    for (int j = 0; j < tn; ++j) {
      const float4 s = tile[j];
      float v = neb_d2(c, s);
      smax = fmaxf(smax, s.z);
      if (v < a[K - 1]) {
#pragma unroll
        for (int q = 0; q < K; ++q) {
          const float lo = fminf(a[q], v);
          v = fmaxf(a[q], v);
          a[q] = lo;
        }
      }
    }
  }
  const bool ok = act && !bad && neb_in_range(smax + c.sc);
  const float u = fmaf(NEB_ABS, smax + c.sc, sqrtf(a[K - 1]) * NEB_REL) * NEB_REL;
  int cnt = 0;
  int32_t* o = out + i * k;
  for (int t0 = 0; t0 < n_ref; t0 += NEB_TILE) {
    const int tn = n_ref <= NEB_TILE ? n_ref : neb_tile(tile, rx, ry, n_ref, t0, ox, oy, bad);
    if (!ok) continue;
    for (int j = 0; j < tn; ++j) {
      const float4 s = tile[j];
      const float lim = fmaf(NEB_ABS, s.z + c.sc, u);
      if (neb_d2(c, s) <= lim * lim) {
        if (cnt < k) o[cnt] = t0 + j;
        ++cnt;
      }
    }
  }
  // (a thread alone took three times as long over its candidates as the whole
  // scan, and held its CTA's place: half of the kernel's time)
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  NebCand& w = cand[warp];
  for (unsigned tie = __ballot_sync(0xffffffffu, ok && cnt != k && cnt <= NEB_CAND); tie;
       tie &= tie - 1) {
    const int src = __ffs((int)tie) - 1;
    const NebCell b = neb_share(c, src);
    const float ub = __shfl_sync(0xffffffffu, u, src);
    int n = 0;
    for (int j0 = 0; j0 < n_ref; j0 += 32) {
      bool hit = false;
      if (j0 + lane < n_ref) {
        const float4 s = neb_stn(tile, rx, ry, n_ref, j0 + lane);
        const float lim = fmaf(NEB_ABS, s.z + b.sc, ub);
        hit = neb_d2(b, s) <= lim * lim;
      }
      neb_append(w, hit, j0 + lane, 0, n);
    }
    n = min(n, NEB_CAND);
    __syncwarp();
    for (int e = lane; e < n; e += 32) w.d[e] = dist_f64(b.x, b.y, rx[w.j[e]], ry[w.j[e]]);
    __syncwarp();
    neb_take(w, n, k, out + (i - lane + src) * k, [&](int e) {
      int r = 0;
      for (int f = 0; f < n; ++f) r += neb_less(w.d[f], f, w.d[e], e);
      return r;
    });
    __syncwarp();
  }
  if (act && (!ok || cnt > NEB_CAND)) neb_nrst_exact(c, rx, ry, n_ref, k, o);
}

// a station's pie by the reference's rules in FP64
__device__ __noinline__ int neb_pie_f64(double x, double y, double rx, double ry, int n_pies) {
  const double xd = rx - x, yd = ry - y;
  const double two_pi = 2.0 * SPI_PI;
  double ang;
  if (xd == 0.0) {
    ang = 0.0;
  } else {
    ang = atan(yd / xd);
    if (xd < 0.0 && yd > 0.0)
      ang = SPI_PI + ang;
    else if (xd < 0.0 && yd < 0.0)
      ang = SPI_PI + ang;
    else if (xd > 0.0 && yd < 0.0)
      ang = two_pi + ang;
  }
  const int p = (int)(ang * (double)n_pies / two_pi);
  return min(max(p, 0), n_pies - 1);
}
// The same from FP32 where the direction is clear of the axes and of the
// pies' edges by more than its error (coordinates' error over the distance,
// atan2f's few ulp), else in FP64.
__device__ __forceinline__ int neb_pie(const NebCell& c, float4 s, const double* rx,
                                       const double* ry, int j, int n_pies, float d2) {
  const float ex = s.x - c.xc, ey = s.y - c.yc;
  const float err = NEB_ABS * (s.z + c.sc);
  const float scale = (float)n_pies * 0.15915494309189535f;  // n_pies / 2 pi
  float ang = atan2f(ey, ex);
  ang = ang < 0.0f ? ang + 6.283185307179586f : ang;
  const float q = ang * scale;
  const float tol = scale * (2.0f * err * rsqrtf(d2) + 4e-6f);
  if (fabsf(ex) > err && fabsf(ey) > err && fabsf(q - rintf(q)) > tol)
    return min((int)q, n_pies - 1);
  return neb_pie_f64(c.x, c.y, rx[j], ry[j], n_pies);
}

// The rule in FP64 over every station.
__device__ __noinline__ void neb_pie_exact(const NebCell& c, const double* rx, const double* ry,
                                           int n_ref, int k, int n_pies, int32_t* out) {
  double pd[NEB_PIE_SLOTS];
  int pi_[NEB_PIE_SLOTS];
  int plen[16];
  for (int p = 0; p < n_pies; ++p) plen[p] = 0;
  for (int j = 0; j < n_ref; ++j) {
    const int p = neb_pie_f64(c.x, c.y, rx[j], ry[j], n_pies);
    neb_insert(pd + p * k, pi_ + p * k, &plen[p], k, dist_f64(c.x, c.y, rx[j], ry[j]), j);
  }
  // the first k by (rank within pie, distance, index)
  int sel[NEB_MAX];
  int ns = 0;
  for (int r = 0; r < k && ns < k; ++r) {
    // this rank's stations, ascending by (distance, index), appended
    double rd[16];
    int ri[16];
    int nr = 0;
    for (int p = 0; p < n_pies; ++p)
      if (plen[p] > r) {
        int q = nr++;
        while (q > 0 && neb_less(pd[p * k + r], pi_[p * k + r], rd[q - 1], ri[q - 1])) {
          rd[q] = rd[q - 1];
          ri[q] = ri[q - 1];
          --q;
        }
        rd[q] = pd[p * k + r];
        ri[q] = pi_[p * k + r];
      }
    for (int q = 0; q < nr && ns < k; ++q) sel[ns++] = ri[q];
  }
  sort_ints(sel, ns);
  for (int q = 0; q < k; ++q) out[q] = q < ns ? sel[q] : -1;
}

// pie: a first scan keeps every pie's R smallest squared FP32 distances
// (shared memory, [pie][rank][thread]; R = k as far as NEB_LISTS values go:
// a destination outside the stations has them all in two or three pies and
// needs many of their ranks); whole ranks are taken while they fit in k, of
// the last one the nearest. Each pie then has a largest distance taken, and
// the second scan writes out the stations up to it plus the rounding's
// bound, in ascending index. Where these are exactly k they are the answer.
// Where they are not, or where the last rank's cut falls between two
// distances closer than the bound, the destination's warp puts the rule to
// the stations of the ranks up to the last one in FP64, a candidate to a
// lane; the destination's thread puts it to every station where the ranks
// kept don't suffice, or the coordinates are out of the bounds' range.
//
// 12 of 270 stations in 8 pies at 20 083 destinations (a warp to a scheduler,
// all latency): 1.6 ms with FP64 angles and lists in local memory, 0.33 with
// undecided destinations left to a thread, 0.21 now.
constexpr int NEB_LISTS = 192;  // values a thread keeps: at most 104 KB a CTA

__global__ __launch_bounds__(NEB_T) void k_neb_pie(const double* __restrict__ dx_,
                                                   const double* __restrict__ dy_,
                                                   int64_t n_dst,
                                                   const double* __restrict__ rx,
                                                   const double* __restrict__ ry, int n_ref,
                                                   int k, int n_pies, int R,
                                                   int32_t* __restrict__ out) {
  __shared__ float4 tile[NEB_TILE];
  __shared__ NebCand cand[NEB_T / 32];
  extern __shared__ float pies[];  // [n_pies][R + 1][NEB_T]
  float* near = pies + threadIdx.x;
  const int R1 = R + 1;  // (slot R: the limits)
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const bool act = i < n_dst;
  const double ox = rx[0], oy = ry[0];
  const NebCell c = neb_cell(dx_, dy_, i, act, ox, oy);
  for (int e = 0; e < n_pies * (R + 1); ++e) near[e * NEB_T] = INFINITY;
  float smax = 0.0f;
  bool bad = false;
  for (int t0 = 0; t0 < n_ref; t0 += NEB_TILE) {
    const int tn = neb_tile(tile, rx, ry, n_ref, t0, ox, oy, bad);
    for (int j = 0; j < tn; ++j) {
      const float4 s = tile[j];
      const float v = neb_d2(c, s);
      smax = fmaxf(smax, s.z);
      float* l = near + neb_pie(c, s, rx, ry, t0 + j, n_pies, v) * (R1 * NEB_T);
      if (v < l[(R - 1) * NEB_T]) {
        int r = R - 1;
        for (; r > 0; --r) {
          const float o = l[(r - 1) * NEB_T];
          if (!(o > v)) break;
          l[r * NEB_T] = o;
        }
        l[r * NEB_T] = v;
      }
    }
  }
  // whole ranks
  int left = k, r = 0;
  bool ok = act && !bad && neb_in_range(smax + c.sc);
  bool in_lists = ok;
  for (;; ++r) {
    int nr = 0;
    if (r < R)
      for (int p = 0; p < n_pies; ++p) nr += near[(p * R1 + r) * NEB_T] < INFINITY;
    if (nr == 0 || nr > left) {
      // (nr == 0: the ranks kept, or the stations, are used up)
      if (nr == 0 && left > 0) ok = in_lists = false;
      break;
    }
    left -= nr;
  }
  const float slack = 2.0f * NEB_ABS * (smax + c.sc);
  // of rank r the nearest left: cut = the largest one taken, next = the
  // smallest one not taken
  float cut = -1.0f, next = INFINITY;
  if (ok && left > 0) {
    for (int q = 0; q <= left; ++q) {
      float m = INFINITY;
      for (int p = 0; p < n_pies; ++p) {
        const float v = near[(p * R1 + r) * NEB_T];
        if (v > cut) m = fminf(m, v);
      }
      if (q < left) cut = m;
      else next = m;
    }
    if (!(sqrtf(next) > sqrtf(cut) * NEB_REL * NEB_REL + 2.0f * slack)) ok = false;
  }
  // each pie's largest distance taken
  for (int p = 0; p < n_pies; ++p) {
    float* l = near + p * (R1 * NEB_T);
    float far = -1.0f;
    for (int e = 0; e < r; ++e) {
      const float v = l[e * NEB_T];
      if (v < INFINITY) far = v;
    }
    if (ok && left > 0 && l[r * NEB_T] <= cut) far = l[r * NEB_T];
    l[R * NEB_T] = far < 0.0f ? -1.0f : fmaf(sqrtf(far) * NEB_REL, NEB_REL, slack);
  }
  int cnt = 0;
  int32_t* o = out + i * k;
  for (int t0 = 0; t0 < n_ref; t0 += NEB_TILE) {
    const int tn = n_ref <= NEB_TILE ? n_ref : neb_tile(tile, rx, ry, n_ref, t0, ox, oy, bad);
    if (!ok) continue;
    for (int j = 0; j < tn; ++j) {
      const float4 s = tile[j];
      const float v = neb_d2(c, s);
      const float lim =
          near[(neb_pie(c, s, rx, ry, t0 + j, n_pies, v) * R1 + R) * NEB_T];
      if (lim >= 0.0f && v <= lim * lim) {
        if (cnt < k) o[cnt] = t0 + j;
        ++cnt;
      }
    }
  }
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  NebCand& w = cand[warp];
  const bool undecided = act && (!ok || cnt != k);
  if (undecided && in_lists)
    // the stations that may be of a rank up to r, or (whole ranks only) of one
    // below it
    for (int p = 0; p < n_pies; ++p) {
      float* l = near + p * (R1 * NEB_T);
      const float v = l[(left > 0 ? r : max(r - 1, 0)) * NEB_T];
      l[R * NEB_T] = v < INFINITY ? fmaf(sqrtf(v) * NEB_REL, NEB_REL, slack) : INFINITY;
    }
  __syncwarp();
  bool done = !undecided;
  for (unsigned tie = __ballot_sync(0xffffffffu, undecided && in_lists); tie; tie &= tie - 1) {
    const int src = __ffs((int)tie) - 1;
    const NebCell b = neb_share(c, src);
    const float* lims = near - lane + src + R * NEB_T;
    int n = 0;
    for (int j0 = 0; j0 < n_ref; j0 += 32) {
      bool hit = false;
      int p = 0;
      if (j0 + lane < n_ref) {
        const float4 s = neb_stn(tile, rx, ry, n_ref, j0 + lane);
        const float v = neb_d2(b, s);
        p = neb_pie(b, s, rx, ry, j0 + lane, n_pies, v);
        const float lim = lims[p * (R1 * NEB_T)];
        hit = v <= lim * lim;
      }
      neb_append(w, hit, j0 + lane, p, n);
    }
    if (n > NEB_CAND) continue;
    if (lane == src) done = true;
    __syncwarp();
    for (int e = lane; e < n; e += 32) w.d[e] = dist_f64(b.x, b.y, rx[w.j[e]], ry[w.j[e]]);
    __syncwarp();
    // the pie becomes the rank in it
    int rank[NEB_CAND / 32];
#pragma unroll
    for (int q = 0; q < NEB_CAND / 32; ++q) {
      const int e = q * 32 + lane;
      rank[q] = 0;
      if (e < n)
        for (int f = 0; f < n; ++f)
          rank[q] += w.key[f] == w.key[e] && neb_less(w.d[f], f, w.d[e], e);
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < NEB_CAND / 32; ++q)
      if (q * 32 + lane < n) w.key[q * 32 + lane] = rank[q];
    __syncwarp();
    neb_take(w, n, k, out + (i - lane + src) * k, [&](int e) {
      int at = 0;
      for (int f = 0; f < n; ++f)
        at += w.key[f] < w.key[e] ||
              (w.key[f] == w.key[e] && neb_less(w.d[f], f, w.d[e], e));
      return at;
    });
    __syncwarp();
  }
  if (!done) neb_pie_exact(c, rx, ry, n_ref, k, n_pies, o);
}

// Rows of neighbour lists into a hash table of row indices (open addressing,
// linear probing; tab: -1 where free, first: the smallest row of a slot's
// list). Rows are compared in full, so a slot is one list whatever its hash.
__global__ __launch_bounds__(256) void k_neb_hash(const int32_t* __restrict__ nb, int64_t n, int k,
                                                  uint32_t mask, int32_t* __restrict__ tab,
                                                  int32_t* __restrict__ first,
                                                  int32_t* __restrict__ slot) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int32_t* a = nb + i * k;
  uint32_t h = 2166136261u;
  for (int q = 0; q < k; ++q) {
    h = (h ^ (uint32_t)a[q]) * 0x9e3779b1u;
    h ^= h >> 15;
  }
  for (uint32_t probe = 0; probe <= mask; ++probe) {  // (half the table is free)
    const uint32_t s = (h + probe) & mask;
    const int32_t other = atomicCAS(tab + s, -1, (int32_t)i);
    bool same = true;
    if (other >= 0 && other != i) {
      const int32_t* b = nb + (int64_t)other * k;
      for (int q = 0; q < k && same; ++q) same = a[q] == b[q];
    }
    if (same) {
      atomicMin(first + s, (int32_t)i);
      slot[i] = (int32_t)s;
      return;
    }
  }
}
__global__ __launch_bounds__(256) void k_neb_first(int64_t n, const int32_t* __restrict__ first,
                                                   const int32_t* __restrict__ slot,
                                                   int32_t* __restrict__ rep) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) rep[i] = first[slot[i]];
}

}  // namespace spi

// 2^p >= 2 n slots
static int64_t neb_slots(int64_t n) {
  int64_t s = 2;
  while (s < 2 * n) s *= 2;
  return s;
}

extern "C" int64_t spi_neb_rep_scratch_bytes(int64_t n) {
  if (n < 0 || n > (int64_t)1 << 30) return -1;
  return (2 * neb_slots(n) + n) * (int64_t)sizeof(int32_t);
}

extern "C" int spi_neb_rep(const int32_t* nb, int64_t n, int32_t k, int32_t* rep, void* scratch,
                           int64_t scratch_bytes, spi_stream_t stream) {
  if (n < 0 || k < 1) return SPI_ERR_ARG;
  if (n > (int64_t)1 << 30) return SPI_ERR_TOO_LARGE;
  if (n == 0) return SPI_OK;
  if (!nb || !rep || !scratch || reinterpret_cast<uintptr_t>(scratch) % 16) return SPI_ERR_ARG;
  if (scratch_bytes < spi_neb_rep_scratch_bytes(n)) return SPI_ERR_WORKSPACE;
  const int64_t slots = neb_slots(n);
  int32_t* tab = static_cast<int32_t*>(scratch);
  int32_t *first = tab + slots, *slot = first + slots;
  cudaStream_t st = (cudaStream_t)stream;
  if (cudaMemsetAsync(tab, 0xff, slots * sizeof(int32_t), st) != cudaSuccess ||
      cudaMemsetAsync(first, 0x7f, slots * sizeof(int32_t), st) != cudaSuccess)
    return SPI_ERR_CUDA;
  const unsigned blocks = (unsigned)((n + 255) / 256);
  spi::k_neb_hash<<<blocks, 256, 0, st>>>(nb, n, k, (uint32_t)(slots - 1), tab, first, slot);
  SPI_LAUNCH_CHECK();
  spi::k_neb_first<<<blocks, 256, 0, st>>>(n, first, slot, rep);
  SPI_LAUNCH_CHECK();
  return SPI_OK;
}

extern "C" int spi_neb_select(int32_t method, const double* dst_x, const double* dst_y,
                              int64_t n_dst, const double* ref_x, const double* ref_y,
                              int32_t n_ref, int32_t n_nebs, int32_t n_pies, int32_t* idxs,
                              spi_stream_t stream) {
  if (n_dst < 0 || n_ref < 1 || n_nebs < 1) return SPI_ERR_ARG;
  if (n_dst == 0) return SPI_OK;
  if (!dst_x || !dst_y || !ref_x || !ref_y || !idxs) return SPI_ERR_ARG;
  const int64_t blocks = (n_dst + spi::NEB_T - 1) / spi::NEB_T;
  if (blocks > 0x7fffffff) return SPI_ERR_TOO_LARGE;
  cudaStream_t st = (cudaStream_t)stream;
  if (method == 1) {
    const int k = n_nebs < n_ref ? n_nebs : n_ref;
    if (k > spi::NEB_MAX) return SPI_ERR_TOO_LARGE;
    auto* f = k <= 8 ? spi::k_neb_nrst<8>
                     : (k <= 16 ? spi::k_neb_nrst<16>
                                : (k <= 32 ? spi::k_neb_nrst<32> : spi::k_neb_nrst<64>));
    f<<<(unsigned)blocks, spi::NEB_T, 0, st>>>(dst_x, dst_y, n_dst, ref_x, ref_y, n_ref, k, idxs);
  } else if (method == 2) {
    if (n_pies < 1 || n_nebs < n_pies || n_ref < n_nebs) return SPI_ERR_ARG;
    if (n_nebs > spi::NEB_MAX || n_pies > 16 || n_pies * n_nebs > spi::NEB_PIE_SLOTS)
      return SPI_ERR_TOO_LARGE;
    int R = n_nebs < spi::NEB_LISTS / n_pies ? n_nebs : spi::NEB_LISTS / n_pies;
    const size_t smem = (size_t)n_pies * (R + 1) * spi::NEB_T * sizeof(float);
    if (!spi::smem_opt_in(spi::k_neb_pie, smem)) return SPI_ERR_CUDA;
    spi::k_neb_pie<<<(unsigned)blocks, spi::NEB_T, smem, st>>>(dst_x, dst_y, n_dst, ref_x, ref_y,
                                                                n_ref, n_nebs, n_pies, R, idxs);
  } else {
    return SPI_ERR_ARG;
  }
  SPI_LAUNCH_CHECK();
  return SPI_OK;
}
