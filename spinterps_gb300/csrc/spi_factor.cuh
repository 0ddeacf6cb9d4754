// What the factorisation files share: a system's view, block reductions, and
// the entry points of each file's launches.
#pragma once
#include "spi_common.cuh"

namespace spi {

constexpr int NB = 32;   // panel width of the blocked factorisations
constexpr int FT = 256;  // threads per factor CTA
constexpr int GA = SPI_MAX_DRIFT + 1;

struct SysView {
  int64_t off;
  int n;
  const int32_t* idx;
  int64_t moff;
};

__device__ __forceinline__ SysView sys_view(const spi_systems_t& sys, int s) {
  SysView v;
  v.off = sys.stn_off[s];
  v.n = (int)(sys.stn_off[s + 1] - v.off);
  v.idx = sys.stn_idx + v.off;
  v.moff = sys.mat_off[s];
  return v;
}

// A system's place in a gated launch: systems with gate[s] == want take
// part (gate NULL: all of them).
struct Gate {
  const int32_t* gate;
  int want;
  __device__ __forceinline__ bool skips(int s) const { return gate && gate[s] != want; }
};

// Lower Cholesky factor of every system in place (spi_chol.cu); status[s]
// receives 0 or the 1-based failing pivot.
template <typename T>
int launch_chol(const spi_systems_t& sys, T* arena, int32_t* status, Gate g, cudaStream_t st);

// Linv = L^-1 in x (x == l: in place), and the condition estimate
// n L_00^2 ||Linv||_F^2: with probes == 0 the norm itself and the strictly
// upper part of x zeroed, with probes == 1 Hutchinson's estimate over fixed
// Rademacher vectors (the strictly upper part of x is left as scratch).
template <typename T>
int launch_trinv(const spi_systems_t& sys, const T* l, T* x, const int32_t* status, double* cond,
                 int probes, Gate g, cudaStream_t st);

// The route of every gated system from its factor's status and condition, the
// exact inverse (k_gj, one CTA each, and the pinv check) where that is off the
// Cholesky path (spi_factor.cu).
int launch_routes(const spi_domain_t& dom, const spi_systems_t& sys, const spi_krige_ws_t& ws,
                  double cond_max, Gate g, cudaStream_t st);

// G, S^-1, 1'G and the steps' dual weights of every system (spi_duals.cu).
int launch_duals(const spi_domain_t& dom, const spi_systems_t& sys, const spi_krige_ws_t& ws,
                 const double* vals, cudaStream_t st);

}  // namespace spi
