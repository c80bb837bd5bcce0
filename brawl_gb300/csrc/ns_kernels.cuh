// ns_kernels.cuh -- device state of a nested-sampling run and its launches.
#pragma once

#include "kernels.cuh"

namespace brawl {

struct NsRun {
  ChainJob job;        // geometry, tables, stream, counters, status
  InitJob init;        // initial_setup quotas and interval bounds
  int8_t* walkers;     // K * n_sites compact configurations
  double* energies;    // K
  uint32_t* rnde;      // K: the jitter word drawn after each initial_setup
  double* limits;      // n_iter ceilings written by the current launch
  int32_t K, n_steps;
  int32_t n_at;        // n_1*n_2*n_3*n_basis*n_species (nested_sampling.f90:82)
  int32_t half;        // int(K / 2.0) in single precision
  int32_t S;           // fixed-point shift of F
  int32_t extra_steps;
  int64_t n_acc;       // accepted steps of the latest walk
  int64_t iter;        // iterations done
  int32_t n_iter;      // iterations of the current launch
  int32_t lazy_cap;    // steps the deferred-energy log holds (>= 1)
  int32_t rounds_cap;  // steps each half of ns_rounds_kernel's log holds
};

// Order-preserving integer key of a double (larger double, larger key).
__device__ __forceinline__ unsigned long long ns_dkey(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

// Fixed-point lower bound of the room under the ceiling: Gdn <= (pred(limit)
// - E) * 2^S, pred(limit) the largest double below it; a step with
// dE + band <= Gdn certainly lands strictly below the ceiling.
__device__ __forceinline__ long long ns_gap_dn(double limit, double E, int S) {
  const double gd = __dsub_rd(nextafter(limit, -__longlong_as_double(0x7ff0000000000000LL)), E);
  const double m = __dsub_rd(gd, __dmul_ru(fabs(gd), 8.881784197001252e-16));  // - |gd| 2^-50
  const double s = ldexp(m, S);
  if (!(s > -9.0e18)) return -0x7fffffffffffffffll;
  if (s > 9.0e18) return 0x7fffffffffffffffll;
  return (long long)floor(s);
}

// Fixed-point upper bound of the ceiling gap: Gup >= (limit - E) * 2^S.
__device__ __forceinline__ long long ns_gap_up(double limit, double E, int S) {
  const double gd = __dsub_rn(limit, E);
  const double m = __dadd_rn(gd, __dmul_rn(fabs(gd), 8.881784197001252e-16));  // + |gd| 2^-50
  const double s = ldexp(m, S);
  if (!(s < 9.0e18)) return 0x7fffffffffffffffll;
  if (s < -9.0e18) return -0x7fffffffffffffffll;
  return (long long)ceil(s);
}

// Shared memory of a run's walks; lazy_cap 0 gives the bytes without the
// deferred-energy log.
uint32_t ns_smem_bytes(const Geom& g, int lazy_cap);
void launch_ns_init(NsRun* d_runs, int n_runs, cudaStream_t stream);
void launch_ns_jitter(NsRun* d_runs, int n_runs, int max_K, cudaStream_t stream);
// max_z: the largest neighbour count of the runs; all_D: every run's
// difference table D is staged (walker_layout's use_D).
void launch_ns_iterate(NsRun* d_runs, int n_runs, uint32_t smem_bytes, int max_z, bool all_D,
                       cudaStream_t stream);

// The walks in rounds of steps (ns_rounds.cu), for runs of at most 65535 sites and
// 512 cells a side whose sites are no neighbours of themselves.
constexpr uint32_t kNsRoundsOwn = 336;  // (layout_room)
uint32_t ns_rounds_smem_bytes(const Geom& g, int cap);
void launch_ns_rounds(NsRun* d_runs, int n_runs, uint32_t smem_bytes, int max_z, cudaStream_t stream);

}  // namespace brawl
