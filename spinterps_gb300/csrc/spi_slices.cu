// FP64 kriging contractions on the tensor cores, as exact products of 8-bit
// slices (the splitting of Ozaki, Ogita, Oishi and Rump, Numer. Algorithms
// 59, 2012), for the FP64 cell pass and for the OK variance of the
// ill-conditioned FP32-tier systems.
//
// Bound before: FP64 issue. |Linv c|^2 takes n^2 / 2 FP64 FMAs per cell and
// GB300 does about 2 per SM and clock, 1800 times fewer than FP16 products
// on the tensor cores.
//
// Every operand is an integer of 63 bits: a right-hand side entry c as
// VA = c 2^62 / (the structures' sills) (spi_fx.cuh, generated in integers), a
// row of Linv, of the dual columns or of the steps' dual weights as
// VB = b 2^(62 - e), 2^e at least the row's largest magnitude. Each is cut
// into 8 balanced digits of 8 bits, VA = sum_i a_i 256^(7 - i), |a_i| <= 128,
// exact in FP16. Products a_i b_j of one level i + j = l share an accumulator:
// |sum| <= 7.2 * 2^14 * 128 < 2^24 over 128 stations (a leading digit is at
// most 80), so its FP32 sums are exact integers, whatever their order. Levels
// 0..7 (36 digit products) are kept; the rest is under 2^-57 of full scale per
// product. After each 128
// stations the eight accumulators are added into a 96-bit integer per
// (cell, row). Rounding happens in the
// operands only, at 2^-63 of the largest entry, where FP64 rounds every
// product and sum. (With 7 digits, 2^-55, the multipliers of 400 stations,
// sums that cancel, were 8.5e-13 off where FP64 is 4.7e-13.)
//
// One persistent CTA per SM; a work item is (system, 128 cells).
//   1. The threads generate the item's right-hand sides into the CTA's slot of
//      global memory (8 bytes per entry; the slots of all CTAs stay in L2 up
//      to n ~ 800), with the nearest station for SK.
//   2. Blocks of 64 rows (the 8 accumulators of 64 columns fill tensor
//      memory): Linv's rows up to their diagonal, then dual columns and
//      steps. Per 16 stations, the threads cut the slot's entries into FP16
//      digits in shared memory, one thread copies the packed row digits (16
//      KB by a bulk copy, packed once per system) and issues 12 MMAs: digit
//      i of the cells against digits 0..7-i of the rows, stacked along N,
//      lands on levels i..7 at once. A ring of SL_ST stages; while a chunk's
//      last MMAs run, the next stages' digits are made.
//   3. The accumulators are drained (lane = cell) into 96-bit sums, SL_RT rows
//      of a cell to a thread (16 working warps, 96 registers a thread); a
//      block's values are squared and summed in 128-bit integers (variance)
//      or scaled to FP64 (duals, estimates), and the cells' sum check,
//      variance and fields are finished from registers.
//
// Measured (GB300, the cell pass alone): 750 stations on 62 500 cells, OK
// with variance 42 -> 2.6 ms, SK 6.8 -> 1.1 ms; EDK, 400 stations, 200 steps
// on 250 000 cells 44.8 -> 3.9 ms; 150 stations, 24 steps on 40 000 cells 2.5
// -> 0.34 ms. The tensor pipe is busy 31% of the time: the digits'
// making, the drains (which hold the MMAs up, the accumulators filling tensor
// memory) and the generation share the rest. Two CTAs per SM with blocks of
// 32 rows measured 12% slower on the variance (twice the digits to make).
//
// Every wait is bounded: on expiry the CTA (all its threads, at the next
// barrier) raises err, waits, again bounded, for its own copies and MMAs,
// frees its tensor memory and returns.
#include "spi_cells.cuh"
#include "spi_fx.cuh"
#include "spi_slices.cuh"
#include "spi_tc.cuh"

namespace spi {

namespace {

constexpr int SL_M = 128;                       // cells per item (MMA M)
constexpr int SL_R = 64;                        // rows per block
constexpr int SL_D = 8;                         // digits
constexpr int SL_LV = 8;                        // levels kept
constexpr int SL_K = 16;                        // stations per stage (one MMA K)
constexpr int SL_KD = 128 / SL_K;               // stages per drain
constexpr int SL_ST = 4;                        // ring stages
constexpr int SL_W = 16;                        // working warps
constexpr int SL_WT = SL_W * 32;
constexpr int SL_T = SL_WT + 64;                // and one each for MMAs and copies
constexpr int SL_RT = SL_R * SL_M / SL_WT;      // rows of a block per working thread
constexpr uint32_t SL_A_SLICE = SL_M * SL_K * 2;             // one digit of the cells
constexpr uint32_t SL_A_BYTES = SL_D * SL_A_SLICE;           // 32 KB
constexpr uint32_t SL_B_BYTES = SL_D * SL_R * SL_K * 2;      // 16 KB, one packed chunk
constexpr uint32_t SL_STAGE = SL_A_BYTES + SL_B_BYTES;
constexpr int SL_CAP = 256;                     // systems per launch
constexpr uint64_t SL_BIAS = 0x8080808080808080ull;
constexpr int64_t SL_BAND = 64ll << (FX_BITS - 54);  // units around the min_vg_val cut taken in FP64

// The launch's device-side header at the start of the scratch.
struct SlHead {
  unsigned long long mn[2], mx[2];  // ordered encodings of the coordinates' range
  unsigned long long bad;           // a coordinate is not finite
  long long place;                  // 4096 minus the finest place of the coordinates
};

// What a launch contracts: the kriging systems of a batch; given right-hand
// sides against the rows of a matrix (the single-neighbourhood classes).
enum SlMode { kKrige, kRows };

// Per-system record.
struct SlSys {
  FxVg vg;
  int use;      // the system takes this path
  int unit;     // a variance row's unit, 2^unit (of y / sill)
};

struct SlArgs {
  spi_domain_t dom;
  spi_systems_t sys;
  spi_krige_ws_t ws;
  const double* vals;
  spi_out_t out;
  double cond_split;
  int32_t* err;
  int want_var;      // variance rows
  int want_vec;      // dual columns and steps, the fields
  int filter;        // 0: every system, 2: not in an FP32 tier, 3: tier 2 (or all candidates)
  int s0, ns;        // the launch's systems
  int rs;            // row records per system
  long pc;           // packed chunks per system
  SlHead* head;
  FxGrid* grid;
  SlSys* rec;        // [n_sys]
  longlong2* sg;     // [n_sys group][max_n16] station grid coordinates
  int sgs;           // their stride
  int32_t* row_e;    // [group][rs] row exponents
  unsigned char* pack;
  unsigned char* slots;
  long slot_bytes;
  SlRows rows;       // (kRows)
};

__device__ __forceinline__ unsigned long long enc(double x) {
  const long long b = __double_as_longlong(x);
  return b < 0 ? ~(unsigned long long)b : (unsigned long long)b | 0x8000000000000000ull;
}
__device__ __forceinline__ double dec(unsigned long long u) {
  return __longlong_as_double((long long)((u >> 63) ? u & 0x7fffffffffffffffull : ~u));
}

// The range of the coordinates of the cells and of the stations in use: those
// of the systems (stn_off, stn_idx), else all. (A gauge without a value may
// have any coordinates.)
__global__ __launch_bounds__(256) void k_sl_range(spi_domain_t dom, const int64_t* stn_off,
                                                  const int32_t* stn_idx, int n_sys, SlHead* h) {
  unsigned long long mn[2] = {~0ull, ~0ull}, mx[2] = {0, 0};
  bool bad = false;
  int place = 4096;
  auto take = [&](double x, double y) {
    bad = bad || !isfinite(x) || !isfinite(y);
    place = min(place, min(fx_place(x), fx_place(y)));
    const unsigned long long a = enc(x), b = enc(y);
    mn[0] = min(mn[0], a);
    mx[0] = max(mx[0], a);
    mn[1] = min(mn[1], b);
    mx[1] = max(mx[1], b);
  };
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < dom.n_cells; i += step)
    take(dom.cell_x[i], dom.cell_y[i]);
  const int64_t used = stn_idx ? stn_off[n_sys] : dom.n_stns;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < used; i += step) {
    const int64_t st = stn_idx ? stn_idx[i] : i;
    take(dom.stn_x[st], dom.stn_y[st]);
  }
  for (int o = 16; o > 0; o >>= 1) place = min(place, __shfl_xor_sync(0xffffffffu, place, o));
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(&h->bad, 1ull);
  if ((threadIdx.x & 31) == 0) atomicMax(&h->place, 4096ll - place);
  for (int d = 0; d < 2; ++d) {
    for (int o = 16; o > 0; o >>= 1) {
      mn[d] = min(mn[d], __shfl_xor_sync(0xffffffffu, mn[d], o));
      mx[d] = max(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], o));
    }
    if ((threadIdx.x & 31) == 0) {
      atomicMin(&h->mn[d], mn[d]);
      atomicMax(&h->mx[d], mx[d]);
    }
  }
}

__device__ __forceinline__ int dual_rows(const SlArgs& A, int route) {
  if (A.sys.kind == SPI_KIND_SK || route == 1) return 1;
  return extra_rows(A.sys.kind, A.dom.n_drift);
}

// The common grid of the range; false where it has none.
__device__ bool sl_grid(const SlHead* h, FxGrid& g) {
  const int place = 4096 - (int)h->place;
  return fx_grid(dec(h->mn[0]), dec(h->mx[0]), dec(h->mn[1]), dec(h->mx[1]), place, g) && !h->bad;
}

// The grid, and which systems of the launch take this path: on the Cholesky
// path (SK: also the exact-inverse path, whose estimates contract the same
// covariances), every structure with a fixed-point form that the grid resolves,
// and in the pass by its filter.
__global__ __launch_bounds__(256) void k_sl_select(SlArgs A) {
  __shared__ FxGrid g;
  __shared__ int ok;
  if (threadIdx.x == 0) {
    ok = sl_grid(A.head, g);
    if (blockIdx.x == 0) *A.grid = g;
  }
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= A.ns) return;
  const int s = A.s0 + i;
  SlSys& r = A.rec[s];
  const int sk = A.sys.kind == SPI_KIND_SK;
  const int route = A.ws.route[s];
  int use = ok && (route == 0 || (sk && route == 1));
  const bool fast = fp32_tier(A.ws, s, A.cond_split, sk);
  if (A.filter == 2) use = use && !fast;
  if (A.filter == 3) use = use && (A.ws.tier ? A.ws.tier[s] == 2 : fast);
  // (a variogram of nuggets alone has no covariances to contract)
  fx_init(r.vg, A.sys.vg[s], sk, A.dom.min_vg_val, g.q);
  if (!r.vg.ok || r.vg.n == 0 || !fx_resolves(A.sys.vg[s], g)) use = 0;
  r.use = use;
  // |y| <= sqrt(sill) for y = Linv c: y / sill in units of 2^unit, 58 bits
  // with 8 times as much room
  int e = 0;
  frexp(1.0 / sqrt(r.vg.sill > 0.0 ? r.vg.sill : 1.0), &e);
  r.unit = e - 55;
}

// A row of the second operand: its first len values, zeros past them.
struct RowRef {
  const double* p;
  int len;
  __device__ __forceinline__ double at(int k) const { return k < len ? p[k] : 0.0; }
};

// The other mode's only "system".
__global__ void k_sl_select_one(SlArgs A) { A.rec[0].use = 1; }

// The row a block's row index names: variance rows first (in blocks), then
// the dual columns and the steps.
template <int MODE>
__device__ __forceinline__ RowRef row_ref(const SlArgs& A, int s, int n, int nvb, int row) {
  if constexpr (MODE == kRows) {
    if (row >= A.rows.m) return {nullptr, 0};
    return {A.rows.inv + (int64_t)row * A.rows.m, n};
  } else {
    const int64_t soff = A.sys.stn_off[s];
    if (row < nvb * SL_R) {
      if (row >= n) return {nullptr, 0};
      return {A.ws.linv_arena + A.sys.mat_off[s] + (int64_t)row * n, row + 1};
    }
    if (!A.want_vec) return {nullptr, 0};
    const int v = row - nvb * SL_R;
    const int nd = dual_rows(A, A.ws.route[s]);
    if (v < nd) return {A.ws.g_cols + soff * GA + (int64_t)v * n, n};
    const int64_t st = A.sys.step_off[s] + (v - nd);
    if (st >= A.sys.step_off[s + 1]) return {nullptr, 0};
    return {A.ws.w_hat + A.sys.val_off[A.sys.steps[st]], n};
  }
}

// Entries per cell of a system.
template <int MODE>
__device__ __forceinline__ int n_entries(const SlArgs& A, int s) {
  if constexpr (MODE == kRows) return A.rows.n;
  else return (int)(A.sys.stn_off[s + 1] - A.sys.stn_off[s]);
}
// Rows besides the variance's.
template <int MODE>
__device__ __forceinline__ int n_vec(const SlArgs& A, int s) {
  if constexpr (MODE == kRows) return A.rows.m;
  else
    return A.want_vec ? dual_rows(A, A.ws.route[s]) +
                            (int)(A.sys.step_off[s + 1] - A.sys.step_off[s])
                      : 0;
}

__device__ __forceinline__ int var_blocks(const SlArgs& A, int n) {
  return A.want_var ? (n + SL_R - 1) / SL_R : 0;
}

// A row's exponent: 2^e >= its largest magnitude. A row with a value that is
// not finite takes its system off this path. Station grid coordinates are
// filled in on the side.
template <int MODE>
__global__ __launch_bounds__(256) void k_sl_rows(SlArgs A) {
  const int i = blockIdx.y, s = A.s0 + i;
  if (!A.rec[s].use) return;
  const int n = n_entries<MODE>(A, s);
  const int nvb = MODE == kKrige ? var_blocks(A, n) : 0;
  const int lane = threadIdx.x & 31;
  if constexpr (MODE == kKrige) {
    const FxGrid g = *A.grid;
    for (int k = blockIdx.x * 256 + threadIdx.x; k < n; k += gridDim.x * 256) {
      const int st = A.sys.stn_idx[A.sys.stn_off[s] + k];
      A.sg[(int64_t)i * A.sgs + k] = longlong2{fx_coord(A.dom.stn_x[st], g.ox, g.q),
                                               fx_coord(A.dom.stn_y[st], g.oy, g.q)};
    }
  }
  for (int row = blockIdx.x * 8 + (threadIdx.x >> 5); row < A.rs; row += gridDim.x * 8) {
    const RowRef p = row_ref<MODE>(A, s, n, nvb, row);
    // the largest biased exponent by the high words
    int mx = 0;
    for (int j = lane; j < p.len; j += 32) mx = max(mx, __double2hiint(p.at(j)) & 0x7fffffff);
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) {
      const int e = (mx >> 20) - 1022;  // |b| < 2^e
      if ((mx >> 20) == 0x7ff) A.rec[s].use = 0;
      A.row_e[(int64_t)i * A.rs + row] = max(e, -900);
    }
  }
}

// 8 biased entries of one row or cell into 8 digits: byte 7 - i of each, as
// FP16 (0x6400 + u is 1024 + u; minus 1152 is u - 128).
__device__ __forceinline__ void digits8(const uint64_t (&v)[8], uint4 (&o)[SL_D]) {
#pragma unroll
  for (int i = 0; i < SL_D; ++i) {
    const int b = SL_D - 1 - i;
    uint32_t w[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const uint32_t x = (uint32_t)(b >= 4 ? v[2 * p] >> 32 : v[2 * p]);
      const uint32_t y = (uint32_t)(b >= 4 ? v[2 * p + 1] >> 32 : v[2 * p + 1]);
      uint32_t t = __byte_perm(x, y, (uint32_t)((b & 3) | ((4 + (b & 3)) << 8)));
      t = (t & 0x00ff00ffu) | 0x64006400u;
      asm("add.rn.f16x2 %0, %1, %2;" : "=r"(w[p]) : "r"(t), "r"(0xe480e480u));
    }
    o[i] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

__device__ __forceinline__ int var_block_of(int chunk) {
  int b = (int)((sqrtf(1.f + 2.f * (float)chunk) - 1.f) * 0.5f);
  while (2 * (b + 1) * (b + 2) <= chunk) ++b;
  while (2 * b * (b + 1) > chunk) --b;
  return b;
}

// Packed row digits: per (block, 16 stations) 512 rows (digit, row) of 16
// FP16 values in the MMA's tile order. Variance block b starts at chunk
// 2 b (b + 1), its stations ending at its last row.
template <int MODE>
__global__ __launch_bounds__(128) void k_sl_pack(SlArgs A) {
  const int i = blockIdx.y, s = A.s0 + i;
  if (!A.rec[s].use) return;
  const int n = n_entries<MODE>(A, s);
  const int k16 = (n + SL_K - 1) / SL_K, nvb = MODE == kKrige ? var_blocks(A, n) : 0;
  const int nvc = nvb ? 2 * (nvb - 1) * nvb + k16 : 0;
  int c = blockIdx.x, blk, kc;
  if (c < nvc) {
    blk = min(var_block_of(c), nvb - 1);
    kc = c - 2 * blk * (blk + 1);
  } else {
    blk = (c - nvc) / k16;
    kc = (c - nvc) - blk * k16;
    if (blk * SL_R >= n_vec<MODE>(A, s)) return;
    blk += nvb;
  }
  const int r = threadIdx.x & 63, k8 = threadIdx.x >> 6, row = blk * SL_R + r;
  const RowRef p = row_ref<MODE>(A, s, n, nvb, row);
  uint64_t v[8];
  const int e = A.row_e[(int64_t)i * A.rs + row];
  const double sc = ldexp(1.0, FX_BITS - e);
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int k = kc * SL_K + k8 * 8 + q;
    v[q] = (uint64_t)__double2ll_rn(p.at(k) * sc) + SL_BIAS;
  }
  uint4 o[SL_D];
  digits8(v, o);
  unsigned char* dst = A.pack + ((int64_t)i * A.pc + c) * SL_B_BYTES;
#pragma unroll
  for (int d = 0; d < SL_D; ++d) {
    const int rr = d * SL_R + r;
    *reinterpret_cast<uint4*>(dst + k8 * (SL_D * SL_R * 16) + (rr >> 3) * 128 + (rr & 7) * 16) =
        o[d];
  }
}

// D (TMEM) = A B (+ D when acc), FP16 operands.
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc,
                                        uint32_t acc) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ constexpr uint32_t f16_idesc(int n) {
  return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(SL_M >> 4) << 24);
}
__device__ __forceinline__ void tc_commit(uint32_t mbar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
      : "memory");
}
// The working warps' barrier, and the same with the disjunction of a flag.
__device__ __forceinline__ void work_sync() {
  asm volatile("barrier.sync 1, %0;" ::"n"(SL_WT) : "memory");
}
__device__ __forceinline__ bool work_or(int x) {
  int r;
  asm volatile(
      "{\n.reg .pred p, q;\nsetp.ne.s32 q, %1, 0;\nbarrier.red.or.pred p, 1, %2, q;\n"
      "selp.s32 %0, 1, 0, p;\n}\n"
      : "=r"(r)
      : "r"(x), "n"(SL_WT)
      : "memory");
  return r != 0;
}

// a b + c in one instruction (a product by a constant power of two would be
// taken apart into 64-bit shifts)
__device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
  long long d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}

struct SlSmem {
  uint64_t tab[256];
  double q[SL_M][GA];  // the duals; before them the parts' candidates and sums of squares
  double cvar[SL_M];
  int okf[SL_M], nnb[SL_M];
  FxVg vg;
  int list[SL_CAP];
  int nact;
  uint64_t afull[SL_ST], bfull[SL_ST], empty[SL_ST], chunk, drained, quit;
  uint32_t tbase;
  int fail, any_bad;
};

// Waits for use number `use` of a barrier to complete; false, with fail set,
// if it does not within the limit or another role has failed.
__device__ __forceinline__ bool sl_wait(uint64_t* bar, int use, int* fail) {
  const uint32_t m = smem_u32(bar), parity = (uint32_t)(use & 1);
  for (long it = 0; it < TC_SPIN; ++it) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(m), "r"(parity)
        : "memory");
    if (done) return true;
    if ((it & 63) == 63 && *(volatile int*)fail) return false;
  }
  atomicExch(fail, 1);
  return false;
}

// One item's walk over its stages: blocks of rows in order, each over its
// stations. The packed chunks lie in the same order.
struct Walk {
  int nvb, nb, k16;  // variance blocks, all blocks, stages of a full row
  __device__ __forceinline__ int stages(int b) const {
    return b < nvb ? min(4 * (b + 1), k16) : k16;
  }
};

// The FP64 kernel's own decision of an entry within SL_BAND of the cut.
__device__ __noinline__ bool cut_f64(const SlArgs& A, int s, int sk, int64_t gc, int st) {
  const double d =
      dist_f64(A.dom.cell_x[gc], A.dom.cell_y[gc], A.dom.stn_x[st], A.dom.stn_y[st]);
  return vg_fill_f64(A.sys.vg[s], d, sk, A.dom.min_vg_val) == 0.0;
}

// A cell's nearest station so far: the squared distance as a monotone key
// (exponent and 55 bits), and whether another lies within 2^-42 of it, where
// the rounded FP64 distances decide.
struct Near {
  unsigned long long best = ~0ull;
  int bj = -1, amb = 0;
  __device__ __forceinline__ void add(FxDist d, int j) {
    const unsigned long long key = fx_key(d);
    merge(key, j, 0);
  }
  __device__ __forceinline__ void merge(unsigned long long key, int j, int a) {
    const bool less = key < best;
    const unsigned long long gap = less ? best - key : key - best;
    amb = gap < 4096 ? 1 : (less ? a : amb);
    best = less ? key : best;
    bj = less ? j : bj;
  }
};

// This thread's share of the item's right-hand sides, two stations at a
// time, into the slot.
template <int CODE, bool TRACK>
__device__ __forceinline__ void sl_gen(const SlArgs& A, const SlSmem& S, const longlong2* sg,
                                       const int32_t* idx, int n, int k16, int s, int64_t gc,
                                       int64_t cx, int64_t cy, int cell, int part,
                                       ulonglong2* slot, Near& nr) {
  const FxVg& f = S.vg;
  const int64_t cut = f.cut, over = f.over;
  const int sk = f.sk;
  for (int p = part; p < k16 * (SL_K / 2); p += SL_WT / SL_M) {
    const int j = 2 * p;
    // (past the last station the same one again, its entry dropped below)
    const longlong2 s0 = sg[min(j, n - 1)], s1 = sg[min(j + 1, n - 1)];
    const FxDist d[2] = {fx_dist(cx, cy, s0.x, s0.y), fx_dist(cx, cy, s1.x, s1.y)};
    int64_t v[2];
    fx_entries<CODE, 2>(f, d, S.tab, v);
    if constexpr (TRACK) {
      if (j < n) nr.add(d[0], j);
      if (j + 1 < n) nr.add(d[1], j + 1);
    }
    if (cut >= 0) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int64_t gap = v[e] - cut;
        bool z = sk ? gap <= 0 : gap >= 0;
        if (gap <= SL_BAND && gap >= -SL_BAND) z = cut_f64(A, s, sk, gc, idx[min(j + e, n - 1)]);
        v[e] = z ? over : v[e];
      }
    }
    ulonglong2 o;
    o.x = (j < n ? (uint64_t)v[0] : 0) + SL_BIAS;
    o.y = (j + 1 < n ? (uint64_t)v[1] : 0) + SL_BIAS;
    slot[(int64_t)p * SL_M + cell] = o;
  }
}

template <bool TRACK, typename... Args>
__device__ __forceinline__ void sl_gen_any(int code, Args&&... a) {
  switch (code) {
    case SPI_VG_EXP:
      sl_gen<SPI_VG_EXP, TRACK>(a...);
      break;
    case SPI_VG_GAU:
      sl_gen<SPI_VG_GAU, TRACK>(a...);
      break;
    case SPI_VG_SPH:
      sl_gen<SPI_VG_SPH, TRACK>(a...);
      break;
    default:
      sl_gen<-1, TRACK>(a...);
  }
}

// 4 biased entries into 8 digits of 4 FP16 values (a byte of each, as
// digits8).
__device__ __forceinline__ void digits4(const uint64_t (&v)[4], uint2 (&o)[SL_D]) {
#pragma unroll
  for (int i = 0; i < SL_D; ++i) {
    const int b = SL_D - 1 - i;
    uint32_t w[2];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const uint32_t x = (uint32_t)(b >= 4 ? v[2 * p] >> 32 : v[2 * p]);
      const uint32_t y = (uint32_t)(b >= 4 ? v[2 * p + 1] >> 32 : v[2 * p + 1]);
      uint32_t t = __byte_perm(x, y, (uint32_t)((b & 3) | ((4 + (b & 3)) << 8)));
      t = (t & 0x00ff00ffu) | 0x64006400u;
      asm("add.rn.f16x2 %0, %1, %2;" : "=r"(w[p]) : "r"(t), "r"(0xe480e480u));
    }
    o[i] = make_uint2(w[0], w[1]);
  }
}

// x 2^(q0 + 1075) as an integer (under 2^63), rounded; by shifts.
__device__ __forceinline__ int64_t scaled_int(double x, int q0) {
  const int64_t b = __double_as_longlong(x);
  const int e = (int)((b >> 52) & 0x7ff);
  const int64_t m = (b & 0xfffffffffffffll) | (e ? 1ll << 52 : 0);
  const int sh = (e ? e : 1) + q0;  // x = m 2^(e - 1075)
  const int64_t v = sh >= 0 ? m << min(sh, 63) : ((m >> min(-sh - 1, 62)) + 1) >> 1;
  return b < 0 ? -v : v;
}
// (h 2^32 + l) 2^e as a double, rounded; by shifts, and by FP64 operations
// only where it leaves the normal range.
__device__ __forceinline__ double scaled_double(long long h, uint32_t l, int e) {
  const bool neg = h < 0;
  uint64_t a = (uint64_t)h;
  uint32_t b = l;
  if (neg) {
    b = 0u - l;
    a = ~a + (l == 0 ? 1 : 0);
  }
  if (a == 0 && b == 0) return 0.0;
  // the top 64 bits, normalised: |value| = m 2^(32 - c)
  const int c = a ? __clzll((long long)a) : 64 + __clz((int)b);
  const uint64_t m = c >= 32 ? (c < 64 ? a << c : 0) | ((uint64_t)b << (c - 32))
                             : (a << c) | ((uint64_t)b >> (32 - c));
  const int f = 1022 + 63 + 32 - c + e;
  if (f < 1 || f > 2044)
    return scalbn(fma((double)h, 4294967296.0, (double)l), e);
  const uint64_t bits = ((uint64_t)f << 52) + (m >> 11) + ((m >> 10) & 1);
  return __longlong_as_double((long long)(bits | (neg ? 0x8000000000000000ull : 0)));
}

// Given right-hand sides' stations, scaled by a power of two per point. S.nnb:
// its exponent, or kNotFinite.
constexpr int kNotFinite = 0x7fffffff;
// Neighbouring lanes take four pairs of entries of a point (64 bytes of its
// row), eight points to a warp (128 bytes of a slot's line); the scaling is
// a shift of the significand.
__device__ __forceinline__ void sl_gen_rows(const SlArgs& A, SlSmem& S, int n, int k16,
                                            int64_t c0, int64_t C, int tid, ulonglong2* slot) {
  constexpr int PARTS = SL_WT / SL_M;
  const int cell = tid / PARTS, part = tid % PARTS;
  const double* r = A.rows.rhs + min(c0 + cell, C - 1) * A.rows.m;
  int mx = 0;
  for (int j = part; j < n; j += PARTS) mx = max(mx, __double2hiint(r[j]) & 0x7fffffff);
  int* km = reinterpret_cast<int*>(&S.q[0][0]);
  km[part * SL_M + cell] = mx;
  work_sync();
  for (int q = 0; q < PARTS; ++q) mx = max(mx, km[q * SL_M + cell]);
  const bool bad = (mx >> 20) == 0x7ff;
  const int e = max((mx >> 20) - 1022, -900);
  if (part == 0) S.nnb[cell] = bad ? kNotFinite : e;
  const int q0 = FX_BITS - e - 1075;
  for (int p = part; p < k16 * (SL_K / 2); p += PARTS) {
    ulonglong2 v{SL_BIAS, SL_BIAS};
    const int j = 2 * p;
    if (j < n && !bad) v.x += (uint64_t)scaled_int(r[j], q0);
    if (j + 1 < n && !bad) v.y += (uint64_t)scaled_int(r[j + 1], q0);
    slot[(int64_t)p * SL_M + cell] = v;
  }
}

template <int MODE, typename OutT>
__global__ __launch_bounds__(SL_T, 1) void k_sl_gemm(SlArgs A, int tiles) {
  extern __shared__ __align__(1024) unsigned char ring[];
  SlSmem& S = *reinterpret_cast<SlSmem*>(ring + SL_ST * SL_STAGE);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&S.tbase)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 32) {
    S.fail = 0;
    for (int q = 0; q < SL_ST; ++q) {
      mbar_init(smem_u32(&S.afull[q]), SL_W);
      mbar_init(smem_u32(&S.bfull[q]), 1);
      mbar_init(smem_u32(&S.empty[q]), 1);
    }
    mbar_init(smem_u32(&S.chunk), 1);
    mbar_init(smem_u32(&S.drained), SL_W);
    mbar_init(smem_u32(&S.quit), 1);
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  if (tid >= 64 && tid < 64 + 256) S.tab[tid - 64] = fx_exp2_entry(tid - 64);
  if (warp == SL_W) {
    // the launch's active systems
    int cnt = 0;
    for (int b = 0; b < A.ns; b += 32) {
      const int u = b + lane < A.ns ? A.rec[A.s0 + b + lane].use : 0;
      const unsigned m = __ballot_sync(0xffffffffu, u != 0);
      if (u) S.list[cnt + __popc(m & ((1u << lane) - 1))] = b + lane;
      cnt += __popc(m);
    }
    if (lane == 0) S.nact = cnt;
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = S.tbase;
  const int items = S.nact * tiles;
  const int64_t C = MODE == kRows ? A.rows.points : A.dom.n_cells;
  const int sk = MODE == kKrige && A.sys.kind == SPI_KIND_SK;
  int g = 0;     // stages of the earlier items (every role counts them alike)
  int nch = 0;   // their chunks (drains)
  int issued = 0;  // copies issued (the copying thread's)
  bool ok = true;

  for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
    const int li = S.list[item / tiles], s = A.s0 + li;
    const int64_t c0 = (int64_t)(item % tiles) * SL_M;
    const int n = n_entries<MODE>(A, s), vecs = n_vec<MODE>(A, s);
    Walk W;
    W.nvb = MODE == kKrige ? var_blocks(A, n) : 0;
    W.k16 = (n + SL_K - 1) / SL_K;
    W.nb = W.nvb + (vecs + SL_R - 1) / SL_R;

    if (warp == SL_W + 1) {
      // ---- copies of the packed rows ----
      if (lane == 0) {
        int f = g;
        const unsigned char* src = A.pack + (int64_t)li * A.pc * SL_B_BYTES;
        for (int b = 0; b < W.nb && ok; ++b)
          for (int k = 0; k < W.stages(b); ++k, ++f, src += SL_B_BYTES) {
            const int st = f % SL_ST;
            if (f >= SL_ST && !(ok = sl_wait(&S.empty[st], f / SL_ST - 1, &S.fail))) break;
            tc_bulk_load(smem_u32(ring + st * SL_STAGE + SL_A_BYTES),
                         reinterpret_cast<const float*>(src), SL_B_BYTES,
                         smem_u32(&S.bfull[st]));
            issued = f + 1;
          }
      }
      ok = __shfl_sync(0xffffffffu, (int)ok, 0);
      for (int b = 0; b < W.nb; ++b) g += W.stages(b);
      continue;
    }
    if (warp == SL_W) {
      // ---- MMAs ----
      if (lane == 0) {
        int f = g, ch = nch;
        for (int b = 0; b < W.nb && ok; ++b) {
          const int ks = W.stages(b);
          for (int k = 0; k < ks; ++k, ++f) {
            const int st = f % SL_ST;
            const bool first = (k % SL_KD) == 0;
            if (first && ch > 0) ok = sl_wait(&S.drained, ch - 1, &S.fail);
            ok = ok && sl_wait(&S.bfull[st], f / SL_ST, &S.fail) &&
                 sl_wait(&S.afull[st], f / SL_ST, &S.fail);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint32_t sa = smem_u32(ring + st * SL_STAGE);
            const uint64_t da = umma_desc(sa, SL_M * 16, 128);
            const uint64_t db = umma_desc(sa + SL_A_BYTES, SL_D * SL_R * 16, 128);
            const uint32_t acc = first ? 0u : 1u;
            // digit i of the cells against digits j .. j + len - 1 of the
            // rows (the descriptors' addresses are in units of 16 bytes)
            auto go = [&](int i, int j, int len, uint32_t a) {
              mma_f16(tmem + (uint32_t)(SL_R * (i + j)), da + (uint64_t)(i * (SL_A_SLICE / 16)),
                      db + (uint64_t)(j * (SL_R / 8) * 8), f16_idesc(SL_R * len), a);
            };
            go(0, 0, 4, acc);
            go(0, 4, 4, acc);
            go(1, 0, 4, 1u);
            go(1, 4, 3, 1u);
            go(2, 0, 3, 1u);
            go(2, 3, 3, 1u);
            go(3, 0, 3, 1u);
            go(3, 3, 2, 1u);
            go(4, 0, 4, 1u);
            go(5, 0, 3, 1u);
            go(6, 0, 2, 1u);
            go(7, 0, 1, 1u);
            tc_commit(smem_u32(&S.empty[st]));
            if (k % SL_KD == SL_KD - 1 || k == ks - 1) {
              tc_commit(smem_u32(&S.chunk));
              ++ch;
            }
          }
        }
      }
      ok = __shfl_sync(0xffffffffu, (int)ok, 0);
      for (int b = 0; b < W.nb; ++b) {
        g += W.stages(b);
        nch += (W.stages(b) + SL_KD - 1) / SL_KD;
      }
      continue;
    }

    // ---- 1. right-hand sides ----
    ulonglong2* slot = reinterpret_cast<ulonglong2*>(A.slots + (long)blockIdx.x * A.slot_bytes);
    const int cell = tid & (SL_M - 1), part = tid >> 7;
    work_sync();  // the previous item is done with the shared state
    int64_t soff = 0, st0 = 0;
    int route = 0, nd = 0, nsteps = 0;
    if constexpr (MODE == kKrige) {
      soff = A.sys.stn_off[s];
      st0 = A.sys.step_off[s];
      nsteps = (int)(A.sys.step_off[s + 1] - st0);
      route = A.ws.route[s];
      nd = dual_rows(A, route);
      if (tid == 0) S.any_bad = 0;
      for (int e = tid; e < (int)(sizeof(FxVg) / 4); e += SL_WT)
        reinterpret_cast<int*>(&S.vg)[e] = reinterpret_cast<const int*>(&A.rec[s].vg)[e];
      work_sync();
    }
    if constexpr (MODE == kRows) {
      sl_gen_rows(A, S, n, W.k16, c0, C, tid, slot);
    } else {
      const int64_t gc = min(c0 + cell, C - 1);
      const FxGrid gr = *A.grid;
      const int64_t cx = fx_coord(A.dom.cell_x[gc], gr.ox, gr.q);
      const int64_t cy = fx_coord(A.dom.cell_y[gc], gr.oy, gr.q);
      const longlong2* sg = A.sg + (int64_t)li * A.sgs;
      const int32_t* idx = A.sys.stn_idx + soff;
      const int code = S.vg.n == 1 ? S.vg.c[0].code : -1;
      Near nr;
      if (sk && A.want_vec) {
        sl_gen_any<true>(code, A, S, sg, idx, n, W.k16, s, gc, cx, cy, cell, part, slot, nr);
        // the parts' candidates, in the order of their stations' parts: an
        // exact tie between parts is ambiguous and goes to the FP64 search
        unsigned long long* kb = reinterpret_cast<unsigned long long*>(&S.q[0][0]);
        int2* kj = reinterpret_cast<int2*>(kb + (SL_WT / SL_M) * SL_M);
        static_assert((SL_WT / SL_M) * SL_M * 16 <= sizeof(S.q), "candidates fit in q");
        kb[tid] = nr.best;
        kj[tid] = make_int2(nr.bj, nr.amb);
        work_sync();
        if (part == 0) {
          for (int q = 1; q < SL_WT / SL_M; ++q)
            if (kj[q * SL_M + cell].x >= 0)
              nr.merge(kb[q * SL_M + cell], kj[q * SL_M + cell].x, kj[q * SL_M + cell].y);
          S.nnb[cell] = nr.amb ? -1 : nr.bj;
        }
      } else {
        sl_gen_any<false>(code, A, S, sg, idx, n, W.k16, s, gc, cx, cy, cell, part, slot, nr);
        if (part == 0) S.nnb[cell] = -1;
      }
    }
    work_sync();

    // ---- 2. the blocks ----
    const int rq = warp >> 2;                  // rows SL_RT * rq .. of a block
    const int dcell = (warp & 3) * 32 + lane;  // this thread's cell in a drain
    const int64_t dg = c0 + dcell;
    const int32_t* row_e = A.row_e + (int64_t)li * A.rs + rq * SL_RT;
    const double sill = MODE == kKrige ? S.vg.sill : 1.0;
    const int unit = MODE == kKrige ? A.rec[s].unit : 0;
    // a row's sum, acc_h 2^32 + acc_l (units of level 7)
    long long acc_h[SL_RT];
    uint32_t acc_l[SL_RT];
    unsigned long long y0 = 0, y1 = 0;  // sum of squares, 128 bits
    double yd = 0.0;  // rows whose value leaves the integers' range
    int total = 0;
    for (int b = 0; b < W.nb; ++b) total += W.stages(b);
    const int fend = g + total;
    int f = g, fb = 0, fk = 0;  // the fill walk, ahead of the drains
    // this thread cuts 4 entries of a stage: stations 4 fp .. of cell fc,
    // neighbouring lanes the two halves of a 16-byte row (their stores then
    // cover shared memory without conflicts)
    const int fc = (warp & 7) * 16 + (lane >> 1), fp = (warp >> 3) * 2 + (lane & 1);
    const ulonglong2* const src = slot + (fp * 2) * SL_M + fc;
    ulonglong2 nx[2];
    auto fetch = [&]() {
      nx[0] = __ldcg(src + fk * (8 * SL_M));
      nx[1] = __ldcg(src + fk * (8 * SL_M) + SL_M);
    };
    unsigned char* const dig =
        ring + (fp >> 1) * (SL_M * 16) + (fc >> 3) * 128 + (fc & 7) * 16 + (fp & 1) * 8;
    auto fill = [&]() {
      const int st = f % SL_ST;
      if (f >= SL_ST) ok = ok && sl_wait(&S.empty[st], f / SL_ST - 1, &S.fail);
      ok = __all_sync(0xffffffffu, ok);  // (a warp's lanes leave together)
      if (!ok) return;
      const uint64_t v[4] = {nx[0].x, nx[0].y, nx[1].x, nx[1].y};
      if (++fk == W.stages(fb)) {
        fk = 0;
        ++fb;
      }
      ++f;
      if (f < fend) fetch();
      uint2 o[SL_D];
      digits4(v, o);
      unsigned char* dst = dig + st * SL_STAGE;
#pragma unroll
      for (int i = 0; i < SL_D; ++i) *reinterpret_cast<uint2*>(dst + i * SL_A_SLICE) = o[i];
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&S.afull[st]))
                     : "memory");
    };
    fetch();
    int done = g;
    for (int b = 0; b < W.nb; ++b) {
      const int ks = W.stages(b);
#pragma unroll
      for (int r = 0; r < SL_RT; ++r) acc_h[r] = acc_l[r] = 0;
      for (int k0 = 0; k0 < ks; k0 += SL_KD, ++nch) {
        // this chunk's stages and, while its last MMAs run, the digits of
        // the next ones
        done += min(SL_KD, ks - k0);
        const int upto = min(done + SL_ST - 1, fend);
        while (f < upto && ok) fill();
        ok = ok && sl_wait(&S.chunk, nch, &S.fail);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t ta = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(rq * SL_RT);
#pragma unroll
        for (int h = 0; h < SL_RT; h += 8) {
          // levels 4..7 of 8 rows, then levels 0..3 above them
          long long lo[8];
          uint32_t r[8];
#pragma unroll
          for (int l = 4; l < SL_LV; ++l) {
            tmem_ld8(ta + (uint32_t)(l * SL_R + h), r);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const int d = __float2int_rn(__uint_as_float(r[q]));
              lo[q] = mad_wide(d, 1 << (8 * (7 - l)), l == 4 ? (long long)acc_l[h + q] : lo[q]);
            }
          }
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            acc_l[h + q] = (uint32_t)lo[q];
            acc_h[h + q] += lo[q] >> 32;
          }
#pragma unroll
          for (int l = 0; l < 4; ++l) {
            tmem_ld8(ta + (uint32_t)(l * SL_R + h), r);
#pragma unroll
            for (int q = 0; q < 8; ++q)
              acc_h[h + q] = mad_wide(__float2int_rn(__uint_as_float(r[q])), 1 << (8 * (3 - l)),
                                      acc_h[h + q]);
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncwarp();
        if (lane == 0)
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&S.drained))
                       : "memory");
      }
      if (work_or(!ok)) {
        ok = false;
        break;
      }
      if constexpr (MODE == kRows) {
        // (b + row) 0 .. of this thread's point
        const int row0 = b * SL_R + rq * SL_RT;
        const int ec = S.nnb[dcell], m = A.rows.m;
        if (dg < C)
#pragma unroll
          for (int h = 0; h < SL_RT; h += 4) {
            // (four rows at a time: their loads overlap, the others' sums keep
            // their registers)
            double y[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
              y[q] = ec == kNotFinite
                         ? __longlong_as_double(0x7ff8000000000000LL)
                         : scaled_double(acc_h[h + q], acc_l[h + q],
                                         ec + row_e[b * SL_R + h + q] - 68);
            for (int k = n; k < m; ++k) {
              const double r = A.rows.rhs[dg * m + k];
              const double* inv = A.rows.inv + (int64_t)(row0 + h) * m + k;
#pragma unroll
              for (int q = 0; q < 4; ++q)
                y[q] = fma(row0 + h + q < m ? __ldg(inv + (int64_t)q * m) : 0.0, r, y[q]);
            }
            double* lam = A.rows.lambdas + dg * n + row0 + h;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int row = row0 + h + q;
              if (row < n) lam[q] = y[q];
              else if (row < m) A.rows.mus[(int64_t)(row - n) * C + dg] = y[q];
            }
          }
        continue;
      }
      if (b < W.nvb) {
        // squares of y / sill in units of 2^unit
#pragma unroll
        for (int q = 0; q < SL_RT; ++q) {
          if (b * SL_R + rq * SL_RT + q < n) {
            const int e = row_e[b * SL_R + q];
            const int sh = unit - e + 68;  // y = (a 2^32 + bl) 2^(e - 68)
            const long long a = acc_h[q];
            const uint32_t bl = acc_l[q];
            const int lim = 26 + sh;       // |a| < 2^lim keeps y under 2^58
            const long long t = lim < 0 ? 1 : (lim > 62 ? 0 : a >> lim);
            if (t == 0 || t == -1) {
              long long y;
              if (sh >= 32) y = sh > 95 ? 0 : a >> (sh - 32);
              else if (sh >= 0) y = (long long)(((unsigned long long)a << (32 - sh)) | (bl >> sh));
              else y = (long long)(((unsigned long long)a << (32 - sh)) |
                                   ((unsigned long long)bl << -sh));
              const unsigned long long u = (unsigned long long)(y < 0 ? -y : y);
              const unsigned long long pl = u * u;
              y0 += pl;
              y1 += __umul64hi(u, u) + (y0 < pl ? 1 : 0);
            } else {
              const double y = scalbn(fma((double)a, 4294967296.0, (double)bl), e - 68 - unit);
              yd = fma(y, y, yd);
            }
          }
        }
        if (b == W.nvb - 1) {
          const double y2 = ((double)y1 * 18446744073709551616.0 + (double)y0) + yd;
          double(*yyp)[SL_M] = reinterpret_cast<double(*)[SL_M]>(&S.q[0][0]);
          yyp[rq][dcell] = scalbn(y2, 2 * unit) * (sill * sill);
          work_sync();
          if (rq == 0) {
            double v = yyp[0][dcell];
            for (int q = 1; q < SL_WT / SL_M; ++q) v += yyp[q][dcell];
            S.cvar[dcell] = v;
            if (!A.want_vec && dg < C) A.ws.cell_yy[(int64_t)s * C + dg] = v;
          }
        }
        continue;
      }
      // ---- 3. dual columns and steps ----
      const int v0 = (b - W.nvb) * SL_R + rq * SL_RT;
      const bool prim = route == 1;
      const int a = sk ? 1 : extra_rows(A.sys.kind, A.dom.n_drift);
      auto value = [&](int q) {
        return scalbn(sill, row_e[b * SL_R + q] - 68) *
               fma((double)acc_h[q], 4294967296.0, (double)acc_l[q]);
      };
      if (b == W.nvb) {
        if (rq == 0)
#pragma unroll
          for (int q = 0; q < GA; ++q) S.q[dcell][q] = q < nd ? value(q) : 0.0;
        work_sync();
        if (tid < SL_M) {
          const int64_t gq = c0 + tid;
          const double q0 = S.q[tid][0];
          double sl = q0, vv = 0.0;
          if (!prim && !sk) {
            const double* Si = A.ws.s_inv + (int64_t)s * GA * GA;
            double nu0 = 0.0;
            for (int k = 0; k < a; ++k) {
              double t = 0.0;
              for (int l = 0; l < a; ++l) {
                const double fl =
                    l == 0 ? 1.0 : (gq < C ? A.dom.cell_drift[(int64_t)(l - 1) * C + gq] : 0.0);
                t += Si[k * GA + l] * (S.q[tid][l] - fl);
              }
              if (k == 0) nu0 = t;
              sl -= A.ws.g_colsum[(int64_t)s * GA + k] * t;
            }
            if (A.want_var) vv = A.ws.shift[s] * sl - S.cvar[tid] + nu0 * q0 - 2.0 * nu0;
          }
          const int okc = isclose_one(sl) ? 1 : 0;
          S.okf[tid] = okc;
          S.cvar[tid] = okc ? vv : 0.0;
          if (!okc && gq < C && S.nnb[tid] < 0) atomicOr(&S.any_bad, 1);
        }
        work_sync();
        if (S.any_bad) {
          for (int cl = warp; cl < SL_M; cl += SL_W) {
            const int64_t gq = c0 + cl;
            if (gq >= C || S.okf[cl] || S.nnb[cl] >= 0) continue;
            const int j = nnb_f64_warp(A.dom, A.sys.stn_idx + soff, n, A.dom.cell_x[gq],
                                       A.dom.cell_y[gq]);
            if (lane == 0) S.nnb[cl] = j;
          }
          work_sync();
        }
      }
      OutT* est_out = reinterpret_cast<OutT*>(A.out.est);
      OutT* var_out = A.want_var ? reinterpret_cast<OutT*>(A.out.var) : nullptr;
      const int okc = S.okf[dcell], nn = S.nnb[dcell];
#pragma unroll
      for (int q = 0; q < SL_RT; ++q) {
        const int vs = v0 + q - nd;
        if (vs >= 0 && vs < nsteps && dg < C) {
          const int j = A.sys.steps[st0 + vs];
          const int64_t row = A.sys.out_row[j];
          double e;
          if (okc) {
            e = value(q);
            if (!sk) {
              const double* bt = A.ws.beta + (int64_t)j * GA;
              e += bt[0];
              for (int k = 1; k < a; ++k) e += bt[k] * A.dom.cell_drift[(int64_t)(k - 1) * C + dg];
            }
          } else {
            e = A.vals[A.sys.val_off[j] + nn];
          }
          est_out[row * C + dg] = cast_out<OutT>(clip_est(e, A.out));
          if (var_out) var_out[row * C + dg] = cast_out<OutT>(S.cvar[dcell]);
        }
      }
    }
    g = fend;
  }
  __syncthreads();
  if (S.fail) {
    if (tid == 0) atomicExch(A.err, 1);
    // what is still in flight, one more bounded wait each: every stage's last
    // copy, and the MMAs, whose completion only a commit of the thread that
    // issued them signals
    if (warp == SL_W + 1 && lane == 0)
      for (int f = max(0, issued - SL_ST); f < issued; ++f)
        mbar_wait_bounded(smem_u32(&S.bfull[f % SL_ST]), (uint32_t)(f / SL_ST) & 1u);
    if (warp == SL_W && lane == 0) {
      tc_commit(smem_u32(&S.quit));
      mbar_wait_bounded(smem_u32(&S.quit), 0);
    }
    __syncthreads();
  }
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

constexpr size_t SL_SMEM = (size_t)SL_ST * SL_STAGE + sizeof(SlSmem);
static_assert(SL_SMEM <= 227 * 1024, "one CTA per SM");

size_t al(size_t x) { return (x + 255) / 256 * 256; }

int n_sms() {
  int dev = 0, v = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 0;
  return v;
}

// Sizes of the scratch's parts.
struct SlPlan {
  int nvb, rs, sgs, k16;
  long pc;
  size_t fixed, per_sys, slot;
  SlPlan(int max_n, int n_sys, int max_vec, bool var, bool vec, int sms) {
    k16 = (max_n + SL_K - 1) / SL_K;
    nvb = var ? (max_n + SL_R - 1) / SL_R : 0;
    const int veb = vec ? (max_vec + SL_R - 1) / SL_R : 0;
    rs = (nvb + veb) * SL_R;
    sgs = k16 * SL_K;
    pc = (nvb ? 2l * (nvb - 1) * nvb + k16 : 0) + (long)veb * k16;
    slot = al((size_t)SL_M * sgs * 8);
    fixed = al(sizeof(SlHead)) + al(sizeof(FxGrid)) + al((size_t)n_sys * sizeof(SlSys)) +
            slot * sms;
    per_sys = al((size_t)sgs * sizeof(longlong2)) + al((size_t)rs * 4) +
              al((size_t)pc * SL_B_BYTES);
  }
};

}  // namespace

int64_t slices_scratch(int max_n, int n_sys, int max_vec, bool var, bool vec) {
  const int sms = n_sms();
  const SlPlan p(max_n, n_sys, max_vec, var, vec, sms > 0 ? sms : 160);
  // the packs of a group of systems at a time, within about 512 MB
  long grp = (long)((512ull << 20) / (p.per_sys ? p.per_sys : 1));
  grp = grp < 8 ? 8 : (grp > SL_CAP ? SL_CAP : grp);
  if (grp > n_sys) grp = n_sys;
  return (int64_t)(p.fixed + p.per_sys * (size_t)grp + 256);
}

int launch_slices(const SlicesCall& c, SlicesDone* done, cudaStream_t st) {
  const int sms = n_sms();
  if (sms <= 0) return SPI_ERR_CUDA;
  const SlPlan p(c.sys.max_n, c.sys.n_sys, c.max_vec, c.want_var, c.want_vec, sms);
  unsigned char* base = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(c.scratch) + 255) / 256 * 256);
  const int64_t room = c.scratch_bytes - (base - static_cast<unsigned char*>(c.scratch)) -
                       (int64_t)p.fixed;
  const int64_t grp0 = room < 0 ? 0 : room / (int64_t)p.per_sys;
  if (grp0 < 1) return SPI_ERR_WORKSPACE;
  const int grp = (int)(grp0 > SL_CAP ? SL_CAP : grp0);
  const int64_t tiles = (c.dom.n_cells + SL_M - 1) / SL_M;
  if (tiles > 0x7fffffff) return SPI_ERR_TOO_LARGE;
  SlArgs A;
  A.dom = c.dom;
  A.sys = c.sys;
  A.ws = c.ws;
  A.vals = c.vals;
  A.out = c.out;
  A.cond_split = c.cond_split;
  A.err = c.err;
  A.want_var = c.want_var;
  A.want_vec = c.want_vec;
  A.filter = c.filter;
  A.rs = p.rs;
  A.pc = p.pc;
  A.sgs = p.sgs;
  A.slot_bytes = (long)p.slot;
  unsigned char* q = base;
  A.head = reinterpret_cast<SlHead*>(q);
  q += al(sizeof(SlHead));
  A.grid = reinterpret_cast<FxGrid*>(q);
  q += al(sizeof(FxGrid));
  A.rec = reinterpret_cast<SlSys*>(q);
  q += al((size_t)c.sys.n_sys * sizeof(SlSys));
  A.slots = q;
  q += p.slot * sms;
  A.sg = reinterpret_cast<longlong2*>(q);
  q += al((size_t)p.sgs * sizeof(longlong2)) * grp;
  A.row_e = reinterpret_cast<int32_t*>(q);
  q += al((size_t)p.rs * 4) * grp;
  A.pack = q;
  *done = SlicesDone{&A.rec[0].use, (int)(sizeof(SlSys) / sizeof(int32_t)), c.err};
  if (cudaMemsetAsync(A.head->mn, 0xff, sizeof(A.head->mn), st) != cudaSuccess ||
      cudaMemsetAsync(A.head->mx, 0, sizeof(SlHead) - sizeof(A.head->mn), st) != cudaSuccess)
    return SPI_ERR_CUDA;
  k_sl_range<<<2 * sms, 256, 0, st>>>(c.dom, c.sys.stn_off, c.sys.stn_idx, c.sys.n_sys, A.head);
  SPI_LAUNCH_CHECK();
  auto kern = c.out.out_f64 ? k_sl_gemm<kKrige, double> : k_sl_gemm<kKrige, float>;
  if (!smem_opt_in(kern, SL_SMEM)) return SPI_ERR_CUDA;
  for (int s0 = 0; s0 < c.sys.n_sys; s0 += grp) {
    A.s0 = s0;
    A.ns = c.sys.n_sys - s0 < grp ? c.sys.n_sys - s0 : grp;
    k_sl_select<<<(A.ns + 255) / 256, 256, 0, st>>>(A);
    k_sl_rows<kKrige><<<dim3((p.rs + 31) / 32, A.ns), 256, 0, st>>>(A);
    k_sl_pack<kKrige><<<dim3((unsigned)p.pc, A.ns), 128, 0, st>>>(A);
    SPI_LAUNCH_CHECK();
    const int64_t items = tiles * A.ns;
    kern<<<(unsigned)(items < sms ? items : sms), SL_T, SL_SMEM, st>>>(A, (int)tiles);
    SPI_LAUNCH_CHECK();
  }
  return SPI_OK;
}

namespace {

// One "system" of n entries and `rows` rows, its parts laid out in the
// scratch.
int one_layout(SlArgs& A, SlPlan& p, int n, void* scratch, int64_t scratch_bytes, int sms) {
  unsigned char* q = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(scratch) + 255) / 256 * 256);
  if (q + p.fixed + p.per_sys > static_cast<unsigned char*>(scratch) + scratch_bytes)
    return SPI_ERR_WORKSPACE;
  A.s0 = 0;
  A.ns = 1;
  A.rs = p.rs;
  A.pc = p.pc;
  A.sgs = p.sgs;
  A.slot_bytes = (long)p.slot;
  A.head = reinterpret_cast<SlHead*>(q);
  q += al(sizeof(SlHead));
  A.grid = reinterpret_cast<FxGrid*>(q);
  q += al(sizeof(FxGrid));
  A.rec = reinterpret_cast<SlSys*>(q);
  q += al(sizeof(SlSys));
  A.slots = q;
  q += p.slot * sms;
  A.sg = reinterpret_cast<longlong2*>(q);
  q += al((size_t)p.sgs * sizeof(longlong2));
  A.row_e = reinterpret_cast<int32_t*>(q);
  q += al((size_t)p.rs * 4);
  A.pack = q;
  return SPI_OK;
}

template <int MODE, typename K>
int one_launch(SlArgs& A, const SlPlan& p, K kern, int64_t points, int sms, cudaStream_t st) {
  const int64_t tiles = (points + SL_M - 1) / SL_M;
  if (tiles > 0x7fffffff) return SPI_ERR_TOO_LARGE;
  if (!smem_opt_in(kern, SL_SMEM)) return SPI_ERR_CUDA;
  k_sl_rows<MODE><<<dim3((p.rs + 31) / 32, 1), 256, 0, st>>>(A);
  k_sl_pack<MODE><<<dim3((unsigned)p.pc, 1), 128, 0, st>>>(A);
  kern<<<(unsigned)(tiles < sms ? tiles : sms), SL_T, SL_SMEM, st>>>(A, (int)tiles);
  SPI_LAUNCH_CHECK();
  return SPI_OK;
}

}  // namespace

namespace {
__global__ void k_fx_scene(const SlHead* h, FxScene* o) { o->ok = sl_grid(h, o->g); }
}  // namespace

int launch_fx_scene(const spi_domain_t& dom, void* scratch, const FxScene** scene,
                    cudaStream_t st) {
  const int sms = n_sms();
  if (sms <= 0) return SPI_ERR_CUDA;
  unsigned char* q = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(scratch) + 255) / 256 * 256);
  SlHead* h = reinterpret_cast<SlHead*>(q);
  FxScene* o = reinterpret_cast<FxScene*>(q + al(sizeof(SlHead)));
  if (cudaMemsetAsync(h->mn, 0xff, sizeof(h->mn), st) != cudaSuccess ||
      cudaMemsetAsync(h->mx, 0, sizeof(SlHead) - sizeof(h->mn), st) != cudaSuccess)
    return SPI_ERR_CUDA;
  k_sl_range<<<2 * sms, 256, 0, st>>>(dom, nullptr, nullptr, 0, h);
  k_fx_scene<<<1, 1, 0, st>>>(h, o);
  SPI_LAUNCH_CHECK();
  *scene = o;
  return SPI_OK;
}

int64_t slices_scratch_one(int n, int rows) {
  const int sms = n_sms();
  const SlPlan p(n, 1, rows, false, true, sms > 0 ? sms : 160);
  return (int64_t)(p.fixed + p.per_sys + 256);
}

int launch_slices_rows(const SlRows& r, void* scratch, int64_t scratch_bytes, int32_t* err,
                       const int32_t** use, cudaStream_t st) {
  const int sms = n_sms();
  if (sms <= 0) return SPI_ERR_CUDA;
  SlPlan p(r.n, 1, r.m, false, true, sms);
  SlArgs A = {};
  if (int rc = one_layout(A, p, r.n, scratch, scratch_bytes, sms)) return rc;
  A.err = err;
  A.rows = r;
  *use = &A.rec[0].use;
  k_sl_select_one<<<1, 1, 0, st>>>(A);
  return one_launch<kRows>(A, p, k_sl_gemm<kRows, double>, r.points, sms, st);
}

}  // namespace spi

using namespace spi;

extern "C" int64_t spi_slices_scratch_bytes(int32_t max_n, int32_t n_sys, int32_t max_steps,
                                            int32_t n_drift, int32_t want_var,
                                            int32_t want_fields) {
  if (max_n < 1 || n_sys < 1 || max_steps < 0 || n_drift < 0) return 0;
  return slices_scratch(max_n, n_sys, 1 + n_drift + max_steps, want_var != 0, want_fields != 0);
}
