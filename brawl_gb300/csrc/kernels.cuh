// kernels.cuh -- launch-side declarations shared by the kernel translation
// units and the C-ABI layer.
#pragma once

#include <cstdint>
#include <vector>
#include <cuda_runtime.h>

#include "chain_engine.cuh"
#include "trial_window.cuh"

namespace brawl {

// Shared-memory layout of one chain's CTA, identical on host and device.
// The int32 region I holds the six axis tables, then F, then (when small
// enough) D.
struct SmemLayout {
  uint32_t mt, V, ents, sstart, I, lat, total;
  uint32_t tab_len[3];        // 2n + 2*kHalo per axis
  int32_t F_off, D_off;       // element offsets in I
  int32_t use_D;
};

__host__ __device__ inline uint32_t align_up(uint32_t x, uint32_t a) { return (x + a - 1) / a * a; }

// Shared memory that kernels hold in variables of their own, beside their layouts:
// a layout has a block's limit less these bytes (layout_room).
constexpr uint32_t kOneWarpOwn = 16;  // metropolis_kernel, metropolis_halo_kernel, ns_iterate_kernel, wl_sweep_kernel
constexpr uint32_t kFieldOwn = 1584;  // metropolis_field_kernel
constexpr uint32_t kRoundsOwn = 544;  // metropolis_rounds_kernel
template <class... Own>
constexpr uint32_t own_bytes() { return ((uint32_t)((sizeof(Own) + 15) / 16 * 16) + ...); }
inline uint32_t layout_room(int limit, uint32_t own) { return (uint32_t)limit - own; }

// Before a launch: the kernel may take all the dynamic shared memory that its own
// variables leave (the same value at every launch, so that a launch from another
// thread never finds less than it needs), at the largest carveout.
inline int dynamic_most(uint32_t own) {
  static const int most = [] {  // (the same on every device that runs this code)
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return v;
  }();
  return (int)layout_room(most, own);
}
#define BRAWL_SHARED(own, ...)                                                                        \
  do {                                                                                                \
    cudaFuncSetAttribute(__VA_ARGS__, cudaFuncAttributeMaxDynamicSharedMemorySize, dynamic_most(own)); \
    BRAWL_CARVEOUT(__VA_ARGS__);                                                                      \
  } while (0)

constexpr uint32_t kMaxDBytes = 12 * 1024;

__host__ __device__ inline SmemLayout smem_layout(const Geom& g, bool lattice_in_smem) {
  SmemLayout L;
  const uint32_t nsp = (uint32_t)g.ns + 1;
  const uint32_t nF = nsp * (uint32_t)g.nsh * nsp;
  const uint32_t nD = nsp * nsp * (uint32_t)g.nsh * nsp;
  L.mt = 0;
  L.V = align_up(L.mt + kMTN * 4, 16);
  L.ents = L.V + (uint32_t)(g.ns * g.ns * g.nsh) * 8;
  L.sstart = L.ents + (uint32_t)g.z * 4;
  L.I = align_up(L.sstart + (uint32_t)(g.nsh + 1) * 2, 16);
  L.tab_len[0] = 2 * (uint32_t)g.n1 + 2 * kHalo;
  L.tab_len[1] = 2 * (uint32_t)g.n2 + 2 * kHalo;
  L.tab_len[2] = 2 * (uint32_t)g.n3 + 2 * kHalo;
  const uint32_t ntab = 2 * (L.tab_len[0] + L.tab_len[1] + L.tab_len[2]);
  L.use_D = nD * 4 <= kMaxDBytes ? 1 : 0;
  L.F_off = (int32_t)ntab;
  L.D_off = (int32_t)(ntab + nF);
  const uint32_t nI = ntab + nF + (L.use_D ? nD : 0);
  L.lat = align_up(L.I + nI * 4, 16);
  L.total = lattice_in_smem ? align_up(L.lat + (uint32_t)g.n_sites, 16) : L.lat;
  return L;
}

// Builds the wrapping and identity axis tables (see AxisTables).
__device__ inline void build_axis_tables(const Geom& g, int32_t* tabs, const uint32_t* tab_len,
                                         int lane, AxisTables& T) {
  // tabs: the start of the int32 region I
  int32_t* base = tabs;
  const int n[3] = {g.n1, g.n2, g.n3};
  const int W[3] = {g.W1, g.W2, g.W3};
  for (int a = 0; a < 3; ++a) {
    const int len = (int)tab_len[a];
    int32_t* wrap = base;
    int32_t* ident = base + len;
    for (int i = lane; i < len; i += 32) {
      const int t = i - kHalo;
      int w = t % W[a];
      w = w < 0 ? w + W[a] : w;
      int vw, vi;
      const int ti = t < 0 ? 0 : (t >= 2 * n[a] ? 2 * n[a] - 1 : t);
      if (a == 0) {
        vw = w >> g.xs;
        vi = ti >> g.xs;
      } else if (a == 1) {
        vw = (w >> g.ys) * g.sy;
        vi = (ti >> g.ys) * g.sy;
      } else {
        vw = w * g.sz;
        vi = ti * g.sz;
      }
      wrap[i] = vw;
      ident[i] = vi;
    }
    if (a == 0) {
      T.tx[0] = wrap;
      T.tx[1] = ident;
    } else if (a == 1) {
      T.ty[0] = wrap;
      T.ty[1] = ident;
    } else {
      T.tz[0] = wrap;
      T.tz[1] = ident;
    }
    base += 2 * len;
  }
}

constexpr int kTbufWords = 2 * kMTN + kRingMirror;  // the ring and its mirror

// Shared memory of a chain of the windowed kernel (metropolis_halo.cu): the
// stream's rings (trial_window.cuh), the positions' records and the lattice
// with its halo (halo_shear.cuh) at fixed places, then the tables.
struct WindowLayout {
  static constexpr uint32_t kRec = GatherRing::kWords * 4;           // kRecRing records of 16 bytes
  static constexpr uint32_t kFlags = kRec + kRecRing * 16;   // and a word of flags each
  static constexpr uint32_t kLat = kFlags + kRecRing * 4;
  uint32_t V, I, D, edelta, ecan, dnbr, sstart, total;
  int32_t Dk;  // bytes of D per species pair: nsh + 1 shells (the last all zero) of ns + 1
};
static_assert(WindowLayout::kRec % 16 == 0 && WindowLayout::kLat % 16 == 0, "16-byte records, lattice and tables");

__host__ __device__ inline WindowLayout window_layout(const Geom& g, const HaloGeom& H) {
  WindowLayout L;
  const uint32_t nsp = (uint32_t)g.ns + 1;
  L.Dk = (int32_t)(((uint32_t)g.nsh + 1) * nsp * 4);
  L.V = align_up(WindowLayout::kLat + (uint32_t)H.kcells, 16);
  L.I = L.V + (uint32_t)(g.ns * g.ns * g.nsh) * 8;
  L.D = L.I + nsp * (uint32_t)g.nsh * nsp * 4;
  L.edelta = L.D + nsp * nsp * (uint32_t)L.Dk;
  L.ecan = L.edelta + (uint32_t)g.z * 4;
  L.dnbr = L.ecan + 2u * (uint32_t)entry_pad(g.z) * 4;
  L.sstart = L.dnbr + 12 * 4;
  L.total = align_up(L.sstart + (uint32_t)(g.nsh + 1) * 2, 16);
  return L;
}

int lane_entries_for(int max_z);

// Sampling reductions of the annealing loop on the device (sampling.cu).
void launch_energy_accumulate(const double* d_e, double* d_sums, double* d_traj, int n, cudaStream_t s);
void launch_acceptance_snapshot(const unsigned long long* d_counters, unsigned long long* d_acc0, int n,
                                cudaStream_t s);
void launch_asro_finish(const unsigned long long* d_counts, const unsigned long long* d_mask, int n_class,
                        int ns, int wc, double* d_rho_out, double* d_rho_sum, cudaStream_t s);
void launch_temperature_stats(int n, const double* d_sums, const unsigned long long* d_counters,
                              const unsigned long long* d_acc0, const double* d_n_atoms, double n_save,
                              double sim_temp, double temp, double n_mc_real, int with_energies,
                              double* d_out, cudaStream_t s);
void launch_asro_stats(int n, int m, const double* d_rho_sum, double n_save, double* d_out, cudaStream_t s);

// Load the code of every kernel variant a translation unit launches (module
// loading is lazy by default; a launch that first loads code waits for the
// kernels already running on the device).
void preload_metropolis_kernels();
void preload_halo_kernels();
void preload_field_kernels();
void preload_ns_kernels();
void preload_ns_rounds_kernels();
void preload_wl_kernels();
void preload_wl_field_kernels();
void preload_wl_enter_kernels();
void preload_lattice_kernels();

// Kernels of the chains that run in shared memory (fcc/bcc).
enum shared_kernel : int {
  kSharedNone = 0,
  kSharedGather = 1,  // the lattice there, neighbours' sums gathered (metropolis_halo.cu)
  kSharedField = 2,   // the sites' fields there too (metropolis_field.cu)
};

// Whether a set of chains that could run with fields should.  A chain with
// fields takes eight warps and its fields' shared memory, so two at most share an
// SM (field_load: the part of an SM it takes); with the lattice alone it is one
// warp, and six or more share one.  Cycles per trial and chain, with fields and
// gathered (GB300, 900 K, four species, six shells): 116 and 572 on bcc 8^3 at
// one chain per SM, 273 and 590 at four, 527 and 658 at eight; 153 and 396 on
// bcc 16^3 (one per SM) at one, 308 and 402 at two, 456 and 407 at three; on fcc
// 8^3 with two species 310 and 368 at four, 456 and 414 at six.  Accepted swaps
// cost the fields most: 6,000 trials of 400 chains of bcc 14^3, five species, two
// shells, from random configurations 2.9 ms with fields and 2.2 gathered at 1500 K,
// 3.9 and 2.6 at 4000 K, where 300 (two on an SM) take 1.7 and 2.2.  So: fields
// while every chain with them has its place at once.
inline double field_load(uint32_t smem) { return 2u * (smem + 1024u) <= 228u * 1024u ? 0.5 : 1.0; }
inline bool fields_pay(double load, int n_sm) { return load <= n_sm; }

// Of two chains on an SM a very hot one (beta_spread as for gather_trials) gathers,
// as it accepts most swaps, unless the sites around a swapped one are so much of its
// lattice that the gather kernel's next trials mostly wait for it.  5,000 trials of
// 300 chains at 0.1, with fields and gathered (ms): bcc 14^3, five species, two shells
// 3.10 and 2.69, bcc 16^3, three and three 2.77 and 2.49, fcc 10^3, four and six 3.40
// and 3.01; at 0.45 2.80 and 2.64, 2.58 and 2.49, 3.11 and 2.92; at 0.8 2.51 and 2.57,
// 2.40 and 2.42, 2.75 and 2.84.  bcc 6^3 with 64 neighbours of 432 sites at 0.1: 2.31
// and 2.83.  One chain on an SM: within 5% of each other at 0.1.
inline bool too_hot_for_fields(double beta_spread, int z, int n_sites) {
  return beta_spread < 0.4 && 16 * z <= n_sites;
}

// Threads per chain with fields: eight warps run the trials; the others share the
// staging and the fields' first sums.  With an SM to itself a chain takes 16 warps,
// four on each scheduler; at 113 registers a block of 16 leaves a second chain no
// place on its SM, and with eight warps two that share one take some 1.2 times as
// long each.  So 16 warps while the chains of all launches, the longest first and one to
// an SM, the next where one has ended, end hardly later than the longest (trials:
// theirs, in any order).  6,000 trials of 100 chains each of
// bcc 6^3, 9^3 and 14^3 at 4000 K: 2.21 ms with 16 warps, 1.48 with eight; two sweeps of
// each (864 to 10,976 trials) 1.88 and 1.96.
int field_threads(std::vector<int64_t>& trials, int n_sm);

// Wang-Landau walkers with fields (wl_field.cu: one to an SM, its registers fill
// one) beside wl_sweep_kernel's, of which two share an SM: while each has an SM to
// itself.  3,000 trials of 152 walkers, fields and sweeps: bcc 6^3 with 8
// neighbours 2.1-2.4 and 2.6-2.9 ms, 8^3 with 50 (nearly all accepted) 3.2-3.5 and
// 3.6, 12^3 with 64 2.7-3.5 and 3.5-3.9, fcc 9^3 with 78 1.4-3.3 and 3.3-4.2.  In a
// second wave it would depend on the acceptance, which is not known beforehand: 304
// walkers 6.3-6.8 and 3.7, 5.1-6.8 and 3.6-4.0, 2.5-6.4 and 3.4-4.3.
inline bool wl_fields_pay(int n_walkers, int n_sm) { return n_walkers <= n_sm; }

// Chains in rounds of trials (metropolis_rounds.cu) where each has an SM to itself
// (its sixteen warps' registers fill one): 152 chains take as long as one, 0.74 ms
// (simple cubic 6^3, 4,000 trials) and 1.0 (8^3, two species), and twice as many
// twice that, where metropolis_kernel, a warp a chain, takes 2.7 and 1.75 for
// either.  So a second wave would still gain where changes of exactly zero are few
// (1.48 against 2.7) and lose where two species make them common (2.0 against 1.75):
// which it is shows only as the chains run, so the line is where no chain waits.
inline bool rounds_pay(int n_chains, int n_sm) { return n_chains <= n_sm; }
// And whether the longest of them pays for half bytes in shared memory, where
// metropolis_kernel leaves the lattice in global memory: 1, 10 and 100 trials of eight
// chains of fcc 40^3 take 74, 76 and 98 us so, and 52, 59 and 123 there.
inline bool nibbles_paid(int64_t n_trials, int n_sites) { return n_trials >= 8 + n_sites / 4096; }
uint32_t round_smem_bytes(const Geom& g, bool nibbles);
void launch_metropolis_rounds(const ChainJob* d_jobs, int n_jobs, bool nibbles, uint32_t smem_bytes, int max_z,
                              cudaStream_t stream);

// Trials per round of the gather kernel, by how hot the chain is: its inverse
// temperature times the spread of its swaps' energy changes.  The hotter, the
// fewer trials a round keeps.  5,000 trials in rounds of one, two and three, a first
// call from random configurations / later ones (ms): 400 chains of bcc 14^3, five
// species, two shells at 0.95: 1.95/1.90, 2.17/2.02 and 2.32/2.15, at 1.3: 1.94/1.84,
// 2.07/1.83 and 2.21/1.86, at 1.5: 1.91/1.80, 2.03/1.74 and 2.13/1.75, at 2:
// 1.90/1.76, 1.96/1.63 and 2.07/1.55; of bcc 24^3, four species, six shells at 1.3:
// 2.31/2.15, 2.56/2.24 and 2.59/2.25, at 2: 2.28/2.09, 2.46/2.06 and 2.47/2.01; of
// fcc 10^3 alike at 1.3: 2.21/2.05, 2.54/2.03 and 2.76/2.09.  Two species order
// earlier: 600 chains of bcc 10^3, six shells at 0.7: 1.78/1.68, 2.07/1.68 and
// 2.27/1.75, at 0.95: 1.74/1.57, 1.93/1.46 and 2.07/1.43.  Four lose to three from
// random configurations (256 of bcc 24^3 at 600 K: 5.9/4.0 and 5.7/4.1).
constexpr int kGatherDefault = 3;
inline int gather_trials(double beta_spread, int ns) {
  return beta_spread < (ns == 2 ? 0.95 : 1.4) ? 1 : beta_spread < 1.5 ? 2 : kGatherDefault;
}

// One launch of them: `count` chains from `first` in launch order, the largest
// shared memory and neighbour count among them, and the trials per
// round of the gather kernel.
struct LaunchGroup {
  int kernel = kSharedNone, depth = kGatherDefault, first = -1, count = 0;
  int threads = 0;   // per chain with fields (field_threads)
  uint32_t smem = 0;
  int max_z = 0;
  int ns = 0;        // species of one of them (field kernel: all are of its field_variant)
  int64_t most = 0;  // the most trials of one chain
};
void launch_metropolis_halo(const ChainJob* d_jobs, int n_jobs, uint32_t smem_bytes, int max_z, int depth,
                            cudaStream_t stream);
void launch_metropolis_field(const ChainJob* d_jobs, int n_jobs, int threads, uint32_t smem_bytes, int max_z, int ns,
                             cudaStream_t stream);
inline void launch_shared_chains(const ChainJob* d_jobs, int n_jobs, const LaunchGroup& G, cudaStream_t stream) {
  if (G.kernel == kSharedField)
    launch_metropolis_field(d_jobs, n_jobs, G.threads, G.smem, G.max_z, G.ns, stream);
  else
    launch_metropolis_halo(d_jobs, n_jobs, G.smem, G.max_z, G.depth, stream);
}

// Metropolis swap trials, one warp (CTA) per chain; max_z is the largest
// neighbour count in the batch (it selects the unrolling of the fast tier).
void launch_metropolis(const ChainJob* d_jobs, int n_jobs, bool lattice_in_smem, bool use_D,
                       uint32_t smem_bytes, int max_z, cudaStream_t stream);

// initial_setup (src/initialise.F90:434-617) on the device, one warp per
// chain.  Per chain: counts[ns] species quotas, lo_w/hi_w[ns] the interval
// bounds in units of 2^-32 (w >= lo_w and w <= hi_w <=> lo <= u <= hi).
// ---------------------------------------------------------------------------
// Site energies in the reference's order: each shell sum starts from 0.0
// and adds V_ex(species, neighbour, shell) in list order; the shell sums are
// added left to right (src/bw_hamiltonian.f90:898-1262, 1712-1910,
// 2059-2106).
// ---------------------------------------------------------------------------
__device__ inline double site_energy_ref(const Geom& g, const int8_t* lat, const double* V,
                                  const uint32_t* ents, const int16_t* sstart, int x, int y,
                                  int z) {
  const int cs = lat[compact_index(g, x, y, z)];
  double total = 0.0;
  for (int sh = 0; sh < g.nsh; ++sh) {
    double e = 0.0;
    for (int k = sstart[sh]; k < sstart[sh + 1]; ++k) {
      int dx, dy, dz, shk;
      unpack_entry(ents[k], dx, dy, dz, shk);
      const int s = lat[neighbour_index(g, x, y, z, dx, dy, dz)];
      e = __dadd_rn(e, V[(cs - 1) + g.ns * ((s - 1) + g.ns * sh)]);
    }
    total = sh == 0 ? e : __dadd_rn(total, e);
  }
  return total;
}

// The doubles of one binade are consecutive in their bits, and a sum that stays in
// the binade rounds its term to a whole number of the binade's ulps, the same
// whatever the sum, unless the term lies halfway between two.  That number for
// term t (bits) and the binade of e (bits; a normal number), in the direction in
// which e's bits grow, modulo 2^64; ok: not halfway, and not past what 63 bits hold.
__host__ __device__ __forceinline__ unsigned long long ulps_of(long long t, long long e, bool& ok) {
  const int et = (int)(t >> 52) & 0x7ff, s = ((int)(e >> 52) & 0x7ff) - (et > 0 ? et : 1);
  const unsigned long long m = (t & 0xfffffffffffffull) | (et > 0 ? 1ull << 52 : 0ull);
  unsigned long long k;
  if (s <= 0) {
    ok = ok && s >= -8;
    k = m << (-s & 15);
  } else {
    const int r = s < 55 ? s : 55;  // (from 55 on it is under half an ulp)
    const unsigned long long half = 1ull << (r - 1);
    ok = ok && (m & (2 * half - 1)) != half;
    k = (m + half) >> r;
  }
  return (t ^ e) < 0 ? 0ull - k : k;
}

// A value passed through: inside the binade of e, and not its first value (a sum
// just under that one rounds more finely).
__host__ __device__ __forceinline__ bool inside_binade(long long b, long long e) {
  return ((b ^ e) >> 52) == 0 && (b & 0xfffffffffffffll) != 0;
}

// total_energy's ordered sum (src/bw_hamiltonian.f90:67-79): energy =
// energy + e(site) over the sites in order, then 0.5 * energy, for one warp.
// Every lane returns the result.
//
// One by one that is a chain of FP64 adds, 64 cycles each.  256 terms at a time
// (eight a lane) are rounded to whole ulps of the sum so far, added as integers,
// and every value passed through is checked to lie in its binade; the terms up to
// the first that leaves it (or lies halfway between two ulps) are done, and that
// one is added by itself.  A sum that keeps leaving its binade (one that stays
// near zero) is added up one by one for a while, longer each time.  256 chains
// of up to 27,648 sites: 1.12 ms one by one, 0.19 ms so.  Up to `few` terms are
// added up one by one: a sum of one chain gains from 128 on, the longest of many
// chains' from 512 (64 chains of 250 and of 432 sites, the whole call, 49 and 60 us
// one by one and 57 and 69 so; of 864 82 and 70 to 83).
constexpr int kFewTerms = 128, kFewTermsOfMany = 512;
__device__ inline double ordered_half_sum_warp(const double* __restrict__ e, int n, int lane, int few = kFewTerms) {
  constexpr int kTerms = 8;
  double energy = 0.0;
  int base = 0, slow = n < few ? n : 32, run = 32;  // terms to add one by one; then how many
  while (base < n) {
    if (slow > 0) {
      // 32 at a time, the next 32 already in flight
      double v = base + lane < n ? e[base + lane] : 0.0;
      for (; slow > 0 && base < n; slow -= 32) {
        const int m = min(32, n - base), next = base + 32 + lane;
        const double v_next = next < n ? e[next] : 0.0;
        for (int k = 0; k < m; ++k) energy = __dadd_rn(energy, __shfl_sync(kFull, v, k));
        v = v_next;
        base += m;
      }
      continue;
    }
    const int first = base + kTerms * lane;
    double v[kTerms];
#pragma unroll
    for (int j = 0; j < kTerms; ++j) v[j] = first + j < n ? e[first + j] : 0.0;
    const long long eb = __double_as_longlong(energy);
    const int ex = (int)(eb >> 52) & 0x7ff;
    unsigned long long k[kTerms], sum = 0;  // (modulo 2^64: past a term that is not settled they may be anything)
    unsigned bad = ex > 60 && ex < 0x7ff ? 0u : 1u;  // bit j: term j is not settled
#pragma unroll
    for (int j = 0; j < kTerms; ++j) {
      bool ok = true;
      k[j] = ulps_of(__double_as_longlong(v[j]), eb, ok);
      sum += k[j];
      bad |= ok ? 0u : 1u << j;
    }
    unsigned long long upto = sum;  // with the lanes before
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long u = __shfl_up_sync(kFull, upto, o);
      upto += lane >= o ? u : 0ull;
    }
    unsigned long long x = (unsigned long long)eb + upto - sum;
    const unsigned long long x0 = x;
#pragma unroll
    for (int j = 0; j < kTerms; ++j) {
      x += k[j];
      bad |= inside_binade((long long)x, eb) ? 0u : 1u << j;
    }
    // the first term that is not settled
    const unsigned lanes = __ballot_sync(kFull, bad != 0);
    const int m = min(kTerms * 32, n - base);
    int at = m;
    if (lanes) {
      const int l = __ffs(lanes) - 1;
      const int j = __ffs(__shfl_sync(kFull, bad, l)) - 1;
      at = min(m, kTerms * l + j);
      // the sum before it, and it
      unsigned long long before = x0;
#pragma unroll
      for (int i = 0; i < kTerms; ++i) before += i < j ? k[i] : 0ull;
      energy = __longlong_as_double((long long)__shfl_sync(kFull, before, l));
      if (at < m) {
        energy = __dadd_rn(energy, e[base + at]);
        base += at + 1;
        slow = at < 16 ? run : 0;
        run = at < 16 ? min(2 * run, 1024) : 32;
        continue;
      }
    } else {
      energy = __longlong_as_double((long long)__shfl_sync(kFull, x, 31));
    }
    base += m;
    run = 32;
  }
  return __dmul_rn(0.5, energy);
}

struct InitJob {
  int8_t* lat;
  uint32_t* rng;
  int32_t n_sites, ns;
  int64_t counts[kMaxSpecies];
  int64_t lo_w[kMaxSpecies];
  int64_t hi_w[kMaxSpecies];
  unsigned long long* counters;
  int32_t* status;
};
void launch_initial_setup(const InitJob* d_jobs, int n_jobs, cudaStream_t stream);

// The site-by-site draw loop of initial_setup for one configuration
// (src/initialise.F90:434-617), on the warp's stream (mt in shared memory at
// position pos).  Every
// word of the stream is one draw: species l + 1 when it falls in the
// interval of species l whose count is below its quota (the last such l,
// as the reference's loop over l leaves it), else no species and the site
// draws again.  Accepted words fill the sites in order.
//
// The warp decides 32 consecutive words at once.  While no word in the
// batch falls in two intervals and no quota can fill inside the batch
// (check + the batch's words of that species <= count), every word's fate
// is known from the counts at the batch's start: the accepted words take
// the next sites in order (a ballot and a prefix count).  A batch where a
// quota fills, or a word sits on two intervals, is decided word by word.
// Returns false when a quota can never be met (guards against a corrupted
// job; the host validates counts).  Lane l keeps species l + 1's interval (as
// 32-bit words; empty: from above to), quota and count: read from memory and
// counted in shared memory for every batch they took 1,600 cycles of it, now 980
// (256 chains of up to 27,648 sites: 0.72 -> 0.44 ms).
__device__ inline bool initial_setup_warp(const InitJob& J, int8_t* lat, uint32_t* mt, int& pos,
                                          unsigned long long& draws, int lane) {
  const int ns = J.ns;
  const int n_sites = J.n_sites;
  const unsigned long long limit = draws + (unsigned long long)n_sites * 4096ull + 1000000ull;
  const unsigned lt_mask = (1u << lane) - 1u;
  uint32_t from = 1u, to = 0u;
  int64_t quota = 0, check = 0;
  if (lane < ns) {
    const int64_t lo = J.lo_w[lane], hi = J.hi_w[lane];
    if (lo <= 0xffffffffll && hi >= 0) {
      from = (uint32_t)(lo < 0 ? 0 : lo);
      to = (uint32_t)(hi > 0xffffffffll ? 0xffffffffll : hi);
    }
    quota = J.counts[lane];
  }
  int site = 0;
  while (site < n_sites) {
    // the next n <= 32 words, none past the end of the current block
    const int avail = kMTN - pos;
    const int n = avail > 0 ? min(32, avail) : 32;
    const uint32_t w = mt_peek(mt, pos, n, lane);
    int cand = 0, hits = 0;
    for (int l = 0; l < ns; ++l) {
      const uint32_t lo = __shfl_sync(kFull, from, l), hi = __shfl_sync(kFull, to, l);  // (all lanes take part)
      const bool in = lane < n && w >= lo && w <= hi;
      cand = in ? l + 1 : cand;
      hits += in;
    }
    // a candidate whose quota is already full is a plain rejection; one
    // whose quota fills inside the batch needs the word-by-word pass
    const unsigned not_full = __ballot_sync(kFull, check < quota) << 1;  // by species
    const bool open = (not_full >> cand) & 1u;
    unsigned acc = __ballot_sync(kFull, open);
    int need_mine = 0;  // lane l < ns: accepted words of species l + 1 in the batch
    for (int l = 0; l < ns; ++l) {
      const int c = __popc(__ballot_sync(kFull, open && cand == l + 1));
      need_mine = lane == l ? c : need_mine;
    }
    const bool fast = __all_sync(kFull, hits <= 1 && !(lane < ns && check + need_mine > quota));
    int consumed = n;
    if (fast) {
      const int r = n_sites - site;
      bool mine = open;
      if (__popc(acc) > r) {
        // the configuration ends inside the batch: its r-th accepted word
        // is the last one consumed (the words after it are not drawn)
        mine = open && __popc(acc & lt_mask) < r;
        acc = __ballot_sync(kFull, mine);
        for (int l = 0; l < ns; ++l) {
          const int c = __popc(__ballot_sync(kFull, mine && cand == l + 1));
          need_mine = lane == l ? c : need_mine;
        }
      }
      if (__popc(acc) == r) consumed = 32 - __clz(acc);
      if (mine) lat[site + __popc(acc & lt_mask)] = (int8_t)cand;
      check += need_mine;
      site += __popc(acc);
    } else {
      for (int k = 0; k < n; ++k) {
        const uint32_t wk = __shfl_sync(kFull, w, k);
        // every species whose interval holds the word and whose quota is
        // open takes the site in turn and uses up one of its quota (a word
        // on the boundary of two intervals uses up both); the last one keeps it
        const bool takes = wk >= from && wk <= to && check < quota;
        const unsigned taken = __ballot_sync(kFull, takes);
        if (taken) {
          check += takes;
          if (lane == 0) lat[site] = (int8_t)(32 - __clz(taken));
          ++site;
          if (site == n_sites) {
            consumed = k + 1;
            break;
          }
        }
      }
    }
    __syncwarp();
    pos += consumed;
    draws += (unsigned long long)consumed;
    if (draws > limit) return false;
  }
  __syncwarp();
  return true;
}

// total_energy (src/bw_hamiltonian.f90:58-81): per-site FP64 energies in the
// reference's order, then the sequential sum over sites in z, y, x order.
struct EnergyJob {
  Geom g;
  const int8_t* lat;
  const double* V;
  const uint32_t* entries;
  const int16_t* shell_start;
  double* site_energy;        // n_sites scratch
  double* out;                // total energy
  int64_t site_offset;        // prefix over chains (for the grid-stride map)
};
void launch_total_energy(const EnergyJob* d_jobs, int n_jobs, int64_t total_sites,
                         cudaStream_t stream);
// Every job's compact lattice (n_sites bytes) copied from src[c].lat to
// dst[c].lat: the snapshot an energy on another stream reads while the
// chains move on.
void launch_lattice_snapshot(const EnergyJob* d_src, const EnergyJob* d_dst, int n_jobs, int max_sites,
                             cudaStream_t stream);

// Site energy of one site (nbr_energy), one thread.
void launch_site_energy(const EnergyJob* d_job, int x, int y, int z, double* out,
                        cudaStream_t stream);

// Conversions between the reference's full doubled grid config(1,2n1,2n2,2n3)
// (x fastest) and the compact occupied-site array.
void launch_pack(const Geom& g, const int8_t* d_grid, int8_t* d_lat, int32_t* d_status,
                 cudaStream_t stream);
void launch_unpack(const Geom& g, const int8_t* d_lat, int8_t* d_grid, cudaStream_t stream);

// The same for every chain of a batch at once: grids concatenated in chain
// order starting at grid_offset[c].
struct GridJob {
  Geom g;
  int8_t* lat;
  int64_t grid_offset;
  int32_t* status;
};
void launch_pack_batch(const GridJob* d_jobs, int n_jobs, int64_t total_cells,
                       const int8_t* d_grids, cudaStream_t stream);
void launch_unpack_batch(const GridJob* d_jobs, int n_jobs, int64_t total_cells, int8_t* d_grids,
                         cudaStream_t stream);
// counts[offsets[c] + (s - 1) * n_sites + i] += 1 for chain c's site i of species s
void launch_alro_add(const GridJob* d_jobs, int n_jobs, double* d_counts, const int64_t* d_offsets,
                     cudaStream_t stream);

}  // namespace brawl
