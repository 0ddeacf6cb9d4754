// The sliced tensor-core contraction (spi_slices.cu) as the cell entry points
// call it.
#pragma once
#include "spi_common.cuh"
#include "spi_fx.cuh"

namespace spi {

// The systems that a sliced contraction has computed, for the kernel that
// computes the others: all of them where one of its waits ran out (*err).
struct SlicesDone {
  const int32_t* use = nullptr;  // use[s * stride] != 0
  int stride = 0;
  const int32_t* err = nullptr;
  __device__ __forceinline__ bool has(int s) const {
    return use && use[(int64_t)s * stride] && !*err;
  }
};

// Right-hand sides rhs [points, m] against the rows of inv [m, m]: the first
// n results to lambdas [points, n], the rest to mus [m - n, points]. The first
// n entries of each, the stations', go through the slices, the others (ones
// and drifts, whose size has nothing to do with the variogram's) through FP64:
// on one scale with them, semivariances of 1e-9 kept 32 bits.
struct SlRows {
  const double* rhs;
  const double* inv;
  int m, n;
  int64_t points;
  double* lambdas;
  double* mus;
};

struct SlicesCall {
  spi_domain_t dom;
  spi_systems_t sys;
  spi_krige_ws_t ws;
  const double* vals;   // (fields)
  spi_out_t out;        // (fields)
  double cond_split;
  int want_var, want_vec;
  int filter;           // 0: every system, 2: not in an FP32 tier, 3: the double-float tier
  int max_vec;          // dual columns plus the most steps of a system
  void* scratch;
  int64_t scratch_bytes;
  int32_t* err;
};

int64_t slices_scratch(int max_n, int n_sys, int max_vec, bool var, bool vec);

// The other contraction's scratch, and its launch: *use != 0 (on the device)
// where it ran, else the caller computes it.
int64_t slices_scratch_one(int n, int rows);
int launch_slices_rows(const SlRows& r, void* scratch, int64_t scratch_bytes, int32_t* err,
                       const int32_t** use, cudaStream_t st);

// The fixed-point grid of a domain's points, at the start of the scratch
// (a few hundred bytes; valid until the scratch is used for something else).
int launch_fx_scene(const spi_domain_t& dom, void* scratch, const FxScene** scene,
                    cudaStream_t st);

// Runs the systems that have a sliced form; done marks them (on the device, in
// stream order), the caller computes the others.
int launch_slices(const SlicesCall& c, SlicesDone* done, cudaStream_t st);

}  // namespace spi
