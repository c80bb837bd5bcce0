// ns_rounds.cu -- the walks of nested sampling (src/nested_sampling.f90:115-206)
// in rounds of eight steps, for runs whose lattice, tables and logs fit in shared
// memory (ns_rounds_smem_bytes): what ns_iterate_kernel does, step for step, on
// the same state.
//
// Eight warps evaluate the next eight steps at once, each on the lattice as the
// steps before its own would leave it if they ended as guessed.  The decisions are
// then taken in order, up to the first that goes against the guess; the steps
// after it are evaluated again.  A step accepts iff the energy stays below the
// ceiling, and a walk under a high ceiling accepts nearly all of them, one under
// a low ceiling nearly none: those two guesses need no more than the last round's
// end.  In between, the steps are evaluated twice, the first time on the lattice
// as it is, which gives a guess for each.
//
// Roles.  Warps 0 to 3 make the stream and its sites (field_engine.cuh's makers),
// warps 4 to 11 are the team, and warps 12 to 15 sum the FP64 energies of the
// accepted steps (lazy_exact.cuh) beside the team's next steps: the log has two
// halves, one being written while the other is summed.
#include "field_engine.cuh"
#include "lazy_exact.cuh"
#include "ns_kernels.cuh"

namespace brawl {

namespace {

constexpr int kNsThreads = 512;
constexpr int kNsTeam = 256;
constexpr int kNsMeet = kNsTeam + 32 * kFieldMakers;
constexpr int kRound = 8;  // steps of a round, one a warp
enum : int { kRejected, kAccepted, kMixed };  // what the steps are guessed to be

// A site of the lattice: its species, and while a round is evaluated the species
// that a step of the round would make of it and that step's number + 1.
constexpr int kSpeciesBits = 4;
static_assert(kMaxSpecies < 1 << kSpeciesBits && kRound < 1 << (16 - 2 * kSpeciesBits), "a site's 16 bits");
constexpr unsigned kSpeciesMask = (1u << kSpeciesBits) - 1;
__device__ __forceinline__ uint16_t pending(int s, int then, int step) {
  return (uint16_t)(s | then << kSpeciesBits | (step + 1) << 2 * kSpeciesBits);
}

struct NsLat {
  const uint16_t* p;
  __device__ __forceinline__ int operator()(int i) const { return p[i] & kSpeciesMask; }
};

}  // namespace

// Shared memory of a run: the stream's rings, a position's site (index;
// coordinates x | y << 10 | z << 20), then V, the axis tables and F, the
// entries, the lattice, the exact step's terms and the log's two halves.
struct NsLayout {
  static constexpr uint32_t kRec = FieldWords::kWords * 4;
  static constexpr uint32_t kV = kRec + kFieldRing * 8;
  uint32_t I, ents, sstart, lat, vbuf, lazy[2], total;
  uint32_t tab_len[3];
  int32_t F_off;  // (in words from I)
};
static_assert(NsLayout::kRec % 8 == 0 && NsLayout::kV % 16 == 0, "8-byte records, tables of doubles");

__host__ __device__ inline NsLayout ns_layout(const Geom& g, int cap) {
  NsLayout L;
  const uint32_t nsp = (uint32_t)g.ns + 1;
  L.I = align_up(NsLayout::kV + (uint32_t)(g.ns * g.ns * g.nsh) * 8, 16);
  L.tab_len[0] = 2 * (uint32_t)g.n1 + 2 * kHalo;
  L.tab_len[1] = 2 * (uint32_t)g.n2 + 2 * kHalo;
  L.tab_len[2] = 2 * (uint32_t)g.n3 + 2 * kHalo;
  L.F_off = (int32_t)(2 * (L.tab_len[0] + L.tab_len[1] + L.tab_len[2]));
  L.ents = L.I + ((uint32_t)L.F_off + nsp * (uint32_t)g.nsh * nsp) * 4;
  L.sstart = L.ents + (uint32_t)g.z * 4;
  L.lat = align_up(L.sstart + (uint32_t)(g.nsh + 1) * 2, 16);
  L.vbuf = align_up(L.lat + 2u * (uint32_t)g.n_sites, 16);
  L.lazy[0] = align_up(L.vbuf + 4u * (uint32_t)g.z * 8, 16);
  L.lazy[1] = L.lazy[0] + (cap > 0 ? lazy_bytes(g, cap) : 0);
  L.total = L.lazy[1] + (cap > 0 ? lazy_bytes(g, cap) : 0);
  return L;
}

uint32_t ns_rounds_smem_bytes(const Geom& g, int cap) { return ns_layout(g, cap).total; }

namespace {

// The team's last logged half on its way to the summing warps, and back.
struct NsShare {
  // the steps' changes in quanta, and whether a step's draws met another's sites
  // (twice: one is read while the next is written)
  int2 res[2][kRound];
  double E, limit;     // the energy before the half's first step
  long long Dlo, Dhi;  // it changed by that many quanta
  int n, half, quit;
  double E_out;        // after the half, with its gaps (gap_up, gap_dn)
  long long gup, gdn;
  int lost, ok;
  double e_new;        // an exact step's
  unsigned long long best[kNsTeam / 32];
  int best_at[kNsTeam / 32];
};
static_assert(own_bytes<FieldEnd, NsShare>() == kNsRoundsOwn, "what the layout leaves room for");

// Barriers besides the makers': the team's (6), a half is handed over (7), it is
// summed (8), the summing warps' own (9).
__device__ __forceinline__ void ns_team_sync() { asm volatile("bar.sync 6, 256;" ::: "memory"); }
__device__ __forceinline__ void sums_begin_arrive() { asm volatile("bar.arrive 7, 384;" ::: "memory"); }
__device__ __forceinline__ void sums_begin_wait() { asm volatile("bar.sync 7, 384;" ::: "memory"); }
__device__ __forceinline__ void sums_end_arrive() { asm volatile("bar.arrive 8, 384;" ::: "memory"); }
__device__ __forceinline__ void sums_end_wait() { asm volatile("bar.sync 8, 384;" ::: "memory"); }
__device__ __forceinline__ void sums_sync() { asm volatile("bar.sync 9, 128;" ::: "memory"); }

// This lane's neighbour entries (lanes 0 to 15: site 1's, 16 to 31: site 2's),
// every 16th: the axis tables' byte
// addresses of the entry's offset, and its shell's of F's rows.
template <int NJ>
struct NsPlan {
  int ex[NJ], ey[NJ], ez[NJ], shp[NJ];
  unsigned valid;
};

template <int NJ>
__device__ __forceinline__ void ns_plan(const Geom& g, const unsigned char* smem, const uint32_t* ents,
                                        const AxisTables& T, int lane, NsPlan<NJ>& P) {
  P.valid = 0;
  const bool sc = g.lattice == kSimpleCubic;
  auto at = [&](const int32_t* tab, int d) {
    return (int)(reinterpret_cast<const unsigned char*>(tab) - smem) + 4 * (d + kHalo);
  };
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const int k = (lane & 15) + 16 * j;
    int dx = 0, dy = 0, dz = 0, sh = 0;
    if (k < g.z) {
      unpack_entry(ents[k], dx, dy, dz, sh);
      P.valid |= 1u << j;
    }
    P.ex[j] = at(T.tx[sc && dx == 0], dx);
    P.ey[j] = at(T.ty[sc && dy == 0], dy);
    P.ez[j] = at(T.tz[sc && dz == 0], dz);
    P.shp[j] = 4 * sh * (g.ns + 1);
  }
}

// The summing warps (`mine` of four).
__device__ __noinline__ void ns_sums(const Geom& g, unsigned char* smem, const NsLayout& L, int cap, NsShare* S, int St,
                                     int mine, int lane) {
  const double* V = reinterpret_cast<const double*>(smem + NsLayout::kV);
  const int16_t* sstart = reinterpret_cast<const int16_t*>(smem + L.sstart);
  volatile NsShare* vs = S;
  for (;;) {
    sums_begin_wait();
    if (vs->quit) return;
    const int n = vs->n;
    const LazyLog LG = lazy_layout(g, smem + L.lazy[vs->half], cap);
    lazy_sites_any<2>(g, V, sstart, LG, n, kFoldNested, 32 * mine + lane, 128);
    sums_sync();
    const double E0 = vs->E, limit = vs->limit;
    const double E = lazy_fold(LG, n, E0, kFoldNested);  // (each of the four)
    if (mine == 0) {
      const double q = ldexp(1.0, -St);
      const int ok = in_quanta(E, E0, vs->Dlo, vs->Dhi, q);
      if (lane == 0) {
        S->E_out = E;
        S->ok = ok;
      }
    } else if (mine == 1) {
      const long long v = ns_gap_up(limit, E, St);
      if (lane == 0) S->gup = v;
    } else if (mine == 2) {
      const long long v = ns_gap_dn(limit, E, St);
      if (lane == 0) S->gdn = v;
    } else {
      const int lost = quanta_bound(E, St) >= (1ll << 51);
      if (lane == 0) S->lost = lost;
    }
    __syncwarp();
    sums_end_arrive();
  }
}

}  // namespace

// The steps depend on one another, so a round's own chain bounds a run: some 2,600
// cycles (the draws 640, the sums over the neighbours 630, the decisions 540, log
// and lattice 480, the stream 220), instruction latency for the most part, for
// seven to eight steps where nearly all are accepted.  ns_iterate_kernel takes
// 1,630 cycles a step, 450 of them waiting for FP64 sums that here run beside the
// steps (a step's 4 z dependent adds are some 100 cycles of the SM's four FP64
// pipes).  16,000 steps of fcc 6^3, five species, three shells: 13.4 ms there,
// 3.4 ms here while all are accepted; at an acceptance of 0.87, 51.6 ms against
// 157.4 ms for 200,000.  64 runs of bcc 5^3, three species, four shells: 28.5 ms
// against 10.0 ms at 0.95, 26.0 against 11.5 at 0.70; bcc 4^3, five shells, at
// 0.53: 53.7 against 23.3.
template <int NJ>
__global__ void __launch_bounds__(kNsThreads, 1) ns_rounds_kernel(NsRun* __restrict__ runs) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ FieldEnd end;
  __shared__ __align__(16) NsShare S;
  NsRun& R = runs[blockIdx.x];
  const ChainJob& J = R.job;
  const Geom g = J.g;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned long long t_start = global_ns();
  const int cap = R.rounds_cap, n = g.n_sites;
  const NsLayout L = ns_layout(g, cap);
  double* V = reinterpret_cast<double*>(smem + NsLayout::kV);
  int32_t* I = reinterpret_cast<int32_t*>(smem + L.I);
  uint32_t* ents = reinterpret_cast<uint32_t*>(smem + L.ents);
  int16_t* sstart = reinterpret_cast<int16_t*>(smem + L.sstart);
  uint16_t* lat = reinterpret_cast<uint16_t*>(smem + L.lat);
  int2* rec = reinterpret_cast<int2*>(smem + NsLayout::kRec);
  {
    const int nsp = g.ns + 1;
    for (int i = tid; i < g.ns * g.ns * g.nsh; i += blockDim.x) V[i] = J.V[i];
    for (int i = tid; i < nsp * g.nsh * nsp; i += blockDim.x) I[L.F_off + i] = J.F[i];
    for (int i = tid; i < g.z; i += blockDim.x) ents[i] = J.entries[i];
    for (int i = tid; i <= g.nsh; i += blockDim.x) sstart[i] = J.shell_start[i];
  }
  AxisTables T;
  build_axis_tables(g, I, L.tab_len, lane, T);  // (every warp, the same values)
  if (tid == 0) {
    end.done = 0;
    S.quit = 0;
  }
  __syncthreads();
  if (warp < kFieldMakers) {
    stream_produce<kNsMeet>(J.rng, smem, &end, warp, lane, [&](const uint32_t* w, int slot) {
      int x, y, z;
      draw_site(g, w[0], w[1], w[2], x, y, z);
      rec[slot] = make_int2(compact_index(g, x, y, z), x | y << 10 | z << 20);
    });
  } else if (warp >= 12) {
    ns_sums(g, smem, L, cap, &S, R.S, warp - 12, lane);
  } else {
    const int mine = warp - kFieldMakers, tt = mine * 32 + lane;  // step `mine` of a round
    const bool second = lane >= 16;                               // its site 2
    NsPlan<NJ> P;
    ns_plan<NJ>(g, smem, ents, T, lane, P);
    const LazyLog log0 = lazy_layout(g, smem + L.lazy[0], cap);
    const int z = g.z;
    const int codes_at = (int)(log0.codes - smem) + (second ? z : 0) + (lane & 15);
    const int spec_at = (int)(reinterpret_cast<unsigned char*>(log0.spec) - smem);
    const int log_bytes = (int)(L.lazy[1] - L.lazy[0]);
    double* vbuf = reinterpret_cast<double*>(smem + L.vbuf);
    const int F_at = (int)L.I + 4 * L.F_off, row_bytes = 4 * g.nsh * (g.ns + 1);
    auto word = [&](int at) { return *reinterpret_cast<const int32_t*>(smem + at); };
    const uint32_t* tw = reinterpret_cast<const uint32_t*>(smem) + FieldWords::kTwAt;
    const int K = R.K, half_K = R.half, St = R.S, band = J.band;
    int extra_steps = R.extra_steps;
    long long n_acc = R.n_acc, it = R.iter;
    unsigned long long c_steps = 0, c_acc = 0;
    unsigned c_exact = 0;
    int status = kStatusOk;
    unsigned n_win = 0;  // windows of the stream passed
    int o = 0;           // the next word's place in the window
    unsigned have = 0;   // the last part waited for
    int flip = 0;        // the results in use
    int mode = kAccepted;
    // k <= 96 words on; the next 96 positions' records are at hand
    auto advance = [&](int k) {
      o += k;
      const unsigned before = n_win / kFieldMakers;
      n_win += (unsigned)(o >> 5);
      o &= kWin - 1;
      if (n_win / kFieldMakers != before) used_arrive<kNsMeet>((int)(before & 1u));
      if ((n_win + 3) / kFieldMakers != have) {
        ++have;
        made_wait<kNsMeet>((int)(have & 1u));
      }
    };
    made_wait<kNsMeet>(0);
    for (int li = 0; li < R.n_iter && status == kStatusOk; ++li) {
      ++it;
      // maxloc: first index of the largest energy
      unsigned long long best = 0;
      int at = 0x7fffffff;
      for (int w = tt; w < K; w += kNsTeam) {
        const unsigned long long k = ns_dkey(R.energies[w]);
        if (k > best || (k == best && w < at)) {
          best = k;
          at = w;
        }
      }
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) {
        const unsigned long long ok = __shfl_xor_sync(kFull, best, d);
        const int oi = __shfl_xor_sync(kFull, at, d);
        if (ok > best || (ok == best && oi < at)) {
          best = ok;
          at = oi;
        }
      }
      if (lane == 0) {
        S.best[mine] = best;
        S.best_at[mine] = at;
      }
      ns_team_sync();
      best = *(volatile unsigned long long*)&S.best[0];
      at = *(volatile int*)&S.best_at[0];
      for (int w = 1; w < kNsTeam / 32; ++w) {
        const unsigned long long k = *(volatile unsigned long long*)&S.best[w];
        const int i = *(volatile int*)&S.best_at[w];
        if (k > best || (k == best && i < at)) {
          best = k;
          at = i;
        }
      }
      const int imax = at;
      const double limit = R.energies[imax];
      if (tt == 0) R.limits[li] = limit;
      // adaptive extra steps (nested_sampling.f90:129-144)
      if (half_K > 0 && (it % half_K) == 0) {
        if (((float)n_acc < (float)R.n_at * 0.05f) && (extra_steps < R.n_steps * 100)) extra_steps += R.n_steps;
      }
      // clone: irnd = ceiling(rnd * K), 0 only when rnd == 0 (clamped to 1)
      const uint32_t wr = tw[(n_win % (FieldWords::kTw / kWin)) * kWin + o];
      advance(1);
      int irnd = (int)(((unsigned long long)wr * (unsigned long long)K + 0xffffffffull) >> 32);
      if (irnd < 1) irnd = 1;
      const int8_t* src = R.walkers + (size_t)(irnd - 1) * n;
      for (int i = tt; i < n; i += kNsTeam) lat[i] = (uint16_t)src[i];
      // E: the walker's exact energy before the half handed over (or, with none,
      // before the one being written); after the n_log steps of the latter it has
      // changed by D quanta, give or take band for each and a rounding each.  A
      // step is certainly rejected from tr quanta on, accepted up to ta.
      double E = R.energies[irnd - 1];
      int n_log = 0, half = 0;
      long long D = 0, tr = 0, ta = 0;
      bool out = false;  // a half is handed over
      auto gaps = [&](long long gup, long long gdn, int lost) {
        gup = max(min(gup, 1ll << 62), -(1ll << 62));
        gdn = max(min(gdn, 1ll << 62), -(1ll << 62));
        // (past 2^51 quanta an update may round by more than one: nothing is
        // settled)
        const long long per = (long long)n_log * (band + 1);
        tr = lost ? 1ll << 62 : gup - (D - per) + band;
        ta = lost ? -(1ll << 62) : gdn - (D + per) - band;
      };
      auto rebase = [&]() {
        gaps(ns_gap_up(limit, E, St), ns_gap_dn(limit, E, St), quanta_bound(E, St) >= (1ll << 51));
      };
      auto take_back = [&]() {
        if (!out) return;
        sums_end_wait();
        const volatile NsShare* vs = &S;
        E = vs->E_out;
        if (!vs->ok) status = kStatusBandViolated;
        out = false;
        gaps(vs->gup, vs->gdn, vs->lost);
      };
      auto hand_over = [&]() {
        take_back();
        if (n_log == 0) return;
        if (tt == 0) {
          const long long per = (long long)n_log * (band + 1);
          S.E = E;
          S.limit = limit;
          S.Dlo = D - per;
          S.Dhi = D + per;
          S.n = n_log;
          S.half = half;
        }
        __syncwarp();
        sums_begin_arrive();
        out = true;
        half ^= 1;
        n_log = 0;
        D = 0;
      };
      rebase();
      ns_team_sync();
      const long long steps = (long long)R.n_steps + extra_steps;
      long long acc = 0;           // accepted steps
      bool carry = false;          // site 1 is drawn, site 2 not yet found
      int c_site = 0, c_xyz = 0;   // that site
      int tries = 0;
      // every draw takes three words: lane l has the site of the l-th next one
      // (with a carried site 1: that one, then the next ones)
      int2 site;
      auto fetch = [&]() {
        const unsigned r0 = n_win * kWin + (unsigned)o - (carry ? 3u : 0u);
        site = rec[(r0 + 3u * lane) & (kFieldRing - 1)];
        if (carry && lane == 0) site = make_int2(c_site, c_xyz);
      };
      fetch();
      long long st = 0;
      while (st < steps && status == kStatusOk) {
        if (n_log + kRound > cap) hand_over();
        const int s_own = lat[site.x] & kSpeciesMask;
        // the lanes of this lane's species; the next one of another
        unsigned same = kFull;
#pragma unroll
        for (int b = 0; b < 3; ++b) {
          const unsigned v = __ballot_sync(kFull, (s_own >> b) & 1);
          same &= (s_own >> b) & 1 ? v : ~v;
        }
        if (g.ns > 7) {
          const unsigned v = __ballot_sync(kFull, (s_own >> 3) & 1);
          same &= (s_own >> 3) & 1 ? v : ~v;
        }
        const int to = __ffs(~same & (0xfffffffeu << lane)) - 1;  // site 2's lane, or -1
        // the step after the one that starts here, after two, after four (32 and
        // more: past the draws looked at)
        auto jump = [&](int n, int at) {
          const int v = __shfl_sync(kFull, n, at & 31);
          return at < 32 ? v : 63;
        };
        const int n1 = to < 0 ? 63 : to + 1;
        const int n2 = jump(n1, n1), n4 = jump(n2, n2);
        // lane j: step j's start, its site 2's lane, the sites and their species
        const int j1 = jump(n1, 0);
        int start = lane & 1 ? j1 : 0;
        const int j2 = jump(n2, start);
        start = lane & 2 ? j2 : start;
        const int j4 = jump(n4, start);
        start = lane & 4 ? j4 : start;
        const int end_at = jump(n1, start) - 1;
        const bool valid = lane < kRound && end_at < 32 && st + lane < steps;
        const int own = site.x | s_own << 16;
        const int A = __shfl_sync(kFull, own, start & 31), B = __shfl_sync(kFull, own, end_at & 31);
        int nst = __popc(__ballot_sync(kFull, valid));
        if (nst == 0) {
          // none of the draws looked at has another species: on with the same
          // site 1, past the draws of its own, which need no more than their
          // species.  (600 steps that draw one atom of 2,048: 20 ms, 39 where each
          // 31 draws took a round's whole set-up, 29 in ns_iterate_kernel; of 20
          // atoms 1.61, 1.91 and 1.36: a round for every step.)
          c_site = __shfl_sync(kFull, site.x, 0);
          c_xyz = __shfl_sync(kFull, site.y, 0);
          const int s_c = __shfl_sync(kFull, s_own, 0);
          advance(carry ? 93 : 96);
          carry = true;
          for (tries += 31; tries <= 1 << 24; tries += 32) {
            const unsigned r0 = n_win * kWin + (unsigned)o;
            const int next = rec[(r0 + 3u * lane) & (kFieldRing - 1)].x;
            const unsigned other = __ballot_sync(kFull, (lat[next] & kSpeciesMask) != s_c);
            if (other) {
              advance(3 * (__ffs(other) - 1));
              break;
            }
            advance(96);
          }
          if (tries > (1 << 24)) {
            status = kStatusBadSpecies;  // a single species: the reference loops forever
            break;
          }
          fetch();
          continue;
        }
        // ---- this warp's step ------------------------------------------------
        const int my_A = __shfl_sync(kFull, A, mine), my_B = __shfl_sync(kFull, B, mine);
        const int my_lanes = __shfl_sync(kFull, start | end_at << 8, mine);
        const int my_a = my_A & 0xffff, my_b = my_B & 0xffff, my_sa = my_A >> 16, my_sb = my_B >> 16;
        const int xyz = __shfl_sync(kFull, site.y, (second ? my_lanes >> 8 : my_lanes) & 31);
        // this half's site, its species before and after, and the other one
        const int at = second ? my_b : my_a, other = second ? my_a : my_b;
        const int so = second ? my_sb : my_sa, sn = second ? my_sa : my_sb;
        const bool writes = (lane & 15) == 0 && mine < nst;
        unsigned G = mode == kAccepted ? (1u << nst) - 1u : 0u;  // the steps guessed to be accepted
        int code[NJ];
        bool again = mode == kMixed;
        for (;;) {
          if (G) {
            if (writes && ((G >> mine) & 1u)) lat[at] = pending(so, sn, mine);
            ns_team_sync();
          }
          if (mine < nst) {
            const int cx = (xyz & 1023) << 2, cy = (xyz >> 8) & 4092, cz = (xyz >> 18) & 4092;
            const int rowN = F_at + sn * row_bytes, rowO = F_at + so * row_bytes;
            int ni[NJ];
            unsigned s[NJ];
#pragma unroll
            for (int j = 0; j < NJ; ++j) ni[j] = word(P.ex[j] + cx) + word(P.ey[j] + cy) + word(P.ez[j] + cz);
#pragma unroll
            for (int j = 0; j < NJ; ++j) s[j] = lat[ni[j]];
            int dE = 0;
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
              // changed by an earlier step of the round (numbers 1 to mine)
              const bool changed = (s[j] >> 2 * kSpeciesBits) - 1u < (unsigned)mine;
              const int v = (int)((changed ? s[j] >> kSpeciesBits : s[j]) & kSpeciesMask);
              const bool met = ni[j] == other;
              const int t = word(rowN + P.shp[j] + 4 * (met ? so : v)) - word(rowO + P.shp[j] + 4 * v);
              code[j] = v | (met ? kLazyPartner : 0);
              dE += (P.valid >> j) & 1u ? t : 0;
            }
            dE = __reduce_add_sync(kFull, dE);
            int met_at = 0;
            if (G) {
              // Draws of this step at sites that the lattice holds as another's.  One
              // that an earlier step changes: the step has to wait (1).  A site of
              // its own that shows a later step's number: the steps after this one
              // have to wait (2), as which of them share the site is not known.
              const int first = my_lanes & 0xff, last = my_lanes >> 8;
              const unsigned by = (unsigned)lat[site.x] >> 2 * kSpeciesBits;  // 0, or a step + 1
              const bool drawn = lane >= first && lane <= last;
              const unsigned early = __ballot_sync(kFull, drawn && by - 1u < (unsigned)mine);
              const unsigned late = __ballot_sync(kFull, drawn && by > (unsigned)mine + 1u);
              met_at = early ? 1 : (late >> first & 1u) | (late >> last & 1u) ? 2 : 0;
            }
            if (lane == 0) S.res[flip][mine] = make_int2(dE, met_at);
          }
          ns_team_sync();
          if (!again) break;
          // the guess: step by step, with the changes of those accepted
          again = false;
          long long c = 0;
#pragma unroll
          for (int j = 0; j < kRound; ++j) {
            const int v = S.res[flip][j].x;
            const bool yes = j < nst && c + v < tr;
            G |= yes ? 1u << j : 0u;
            c += yes ? v : 0;
          }
          if (!G) break;
          flip ^= 1;
        }
        // ---- the decisions, in order: lane j has step j's ---------------------
        const unsigned all = (1u << nst) - 1u;
        const int2 res = lane < nst ? S.res[flip][lane] : make_int2(0, 0);
        const int d = res.x;
        flip ^= 1;
        bool shared = false;  // a site is two steps'
        if (G) {
          const unsigned wait = __ballot_sync(kFull, res.y == 1) | __ballot_sync(kFull, res.y == 2) << 1;
          shared = wait != 0;
          if (shared) nst = min(nst, __ffs(wait) - 1);  // (never step 0)
        }
        long long c = (G >> lane) & 1u ? d : 0;  // the change with the accepted steps before and this one
        if (G) {
#pragma unroll
          for (int k = 1; k < kRound; k *= 2) {
            const long long v = __shfl_up_sync(kFull, c, k);
            c += lane >= k ? v : 0ll;
          }
        }
        const long long with = (G >> lane) & 1u ? c : c + d;
        const long long pass = (long long)(band + 1) * __popc(G & ((1u << lane) - 1u));
        const unsigned up = __ballot_sync(kFull, lane < nst && with >= tr + pass);
        const unsigned under = __ballot_sync(kFull, lane < nst && with <= ta - pass);
        // the first against the guess, or not settled
        const int first = __ffs(~((under & G) | (up & ~G))) - 1;
        const unsigned yes = (under >> first) & 1u, no = (up >> first) & 1u;
        int done = first + (int)(yes | no);
        unsigned took = (G & ((1u << first) - 1u)) | yes << first;
        if (took) {
          const long long v = __shfl_sync(kFull, yes ? with : c, yes ? first : first - 1);
          const int per = __popc(took) * (band + 1);
          D += v;
          tr += per - v;
          ta -= per + v;
        }
        if (mode == kMixed) mode = G == 0 ? kRejected : G == all ? kAccepted : kMixed;
        else if (first < nst && done < kRound / 2) mode = kMixed;
        bool exact = false;
        if (done == 0) {
          // not settled with the logged steps' interval: their exact energy may
          // settle it
          hand_over();
          take_back();
          done = 1;
          const int d0 = __shfl_sync(kFull, d, 0);
          if (d0 >= tr) {
            // rejected
          } else if (d0 <= ta) {
            took = 1;
            D += d0;
            tr += (long long)band + 1 - d0;
            ta -= (long long)band + 1 + d0;
          } else {
            // the exact step, as the reference takes it (the log is empty)
            ++c_exact;
            exact = true;
            if (mine == 0) {
              SitePair p;
              const int xyz1 = __shfl_sync(kFull, xyz, 0), xyz2 = __shfl_sync(kFull, xyz, 16);
              p.ax = xyz1 & 1023;
              p.ay = (xyz1 >> 10) & 1023;
              p.az = xyz1 >> 20;
              p.bx = xyz2 & 1023;
              p.by = (xyz2 >> 10) & 1023;
              p.bz = xyz2 >> 20;
              p.ai = my_a;
              p.bi = my_b;
              p.sa = my_sa;
              p.sb = my_sb;
              double e_un, e_sw;
              exact_pair_energies_staged(g, NsLat{lat}, V, ents, sstart, p, lane, e_un, e_sw, vbuf);
              if (lane == 0) S.e_new = __dadd_rn(E, __dsub_rn(e_sw, e_un));
            }
            ns_team_sync();
            const double e_new = *(volatile double*)&S.e_new;
            if (e_new < limit) {
              took = 1;
              E = e_new;
              rebase();
            }
          }
        }
        if (took | G) {
          const bool mine_taken = (took >> mine) & 1u;
          if (mine_taken && !exact) {
            const int log_at = half ? log_bytes : 0, row = 2 * (n_log + __popc(took & ((1u << mine) - 1u)));
            const int codes = codes_at + log_at + row * z;
#pragma unroll
            for (int j = 0; j < NJ; ++j)
              if ((P.valid >> j) & 1u) smem[codes + 16 * j] = (unsigned char)code[j];
            if (writes) smem[spec_at + log_at + row + second] = (unsigned char)so;
          }
          const bool put_back = writes && ((G >> mine) & 1u) && !mine_taken;
          if (put_back) lat[at] = (uint16_t)so;
          // (or it would undo a taken step's)
          if (shared) ns_team_sync();
          if (writes && mine_taken) lat[at] = (uint16_t)sn;
        }
        const bool settle = took | G;  // sites have been written
        const int taken = __popc(took);
        if (!exact) n_log += taken;
        acc += taken;
        st += done;
        tries = 0;
        const int words = 3 * __shfl_sync(kFull, end_at, done - 1) + (carry ? 0 : 3);
        carry = false;
        advance(words);
        fetch();
        if (settle) ns_team_sync();
      }
      n_acc = acc;
      c_acc += acc;
      c_steps += st;
      hand_over();
      take_back();
      if (status != kStatusOk) break;
      int8_t* dst = R.walkers + (size_t)imax * n;
      for (int i = tt; i < n; i += kNsTeam) dst[i] = (int8_t)lat[i];
      if (tt == 0) R.energies[imax] = E;
      ns_team_sync();
    }
    if (tt == 0) S.quit = 1;
    __syncwarp();
    sums_begin_arrive();
    // the makers have made, or are making, the part after this one and then wait
    // for this one to be used
    const unsigned part = n_win / kFieldMakers;
    if (have == part) made_wait<kNsMeet>((int)((part + 1) & 1u));
    const unsigned long long words = (unsigned long long)kWin * n_win + (unsigned long long)o;
    if (tt == 0) {
      end.words = words;
      end.done = 1;
    }
    __syncwarp();
    used_arrive<kNsMeet>((int)(part & 1u));
    if (tt == 0) {
      R.extra_steps = extra_steps;
      R.n_acc = n_acc;
      R.iter = it;
      unsigned long long* c = J.counters;
      c[kCntTrials] += c_steps;
      c[kCntEvaluated] += c_steps;
      c[kCntDraws] += words;
      c[kCntAccepted] += c_acc;
      c[kCntExactPath] += c_exact;
      if (status != kStatusOk) *J.status = status;
      if (J.t_ns) *J.t_ns = global_ns() - t_start;
    }
  }
}

template <int NJ>
static void launch_rounds_nj(NsRun* d_runs, int n_runs, uint32_t smem_bytes, cudaStream_t stream) {
  BRAWL_SHARED(kNsRoundsOwn, ns_rounds_kernel<NJ>);
  ns_rounds_kernel<NJ><<<n_runs, kNsThreads, smem_bytes, stream>>>(d_runs);
}

void launch_ns_rounds(NsRun* d_runs, int n_runs, uint32_t smem_bytes, int max_z, cudaStream_t stream) {
  if (n_runs <= 0) return;
  if (max_z <= 32) launch_rounds_nj<2>(d_runs, n_runs, smem_bytes, stream);
  else if (max_z <= 48) launch_rounds_nj<3>(d_runs, n_runs, smem_bytes, stream);
  else if (max_z <= 64) launch_rounds_nj<4>(d_runs, n_runs, smem_bytes, stream);
  else if (max_z <= 96) launch_rounds_nj<6>(d_runs, n_runs, smem_bytes, stream);
  else launch_rounds_nj<11>(d_runs, n_runs, smem_bytes, stream);
}

void preload_ns_rounds_kernels() {
  cudaFuncAttributes a;
  cudaFuncGetAttributes(&a, ns_rounds_kernel<2>);
  cudaFuncGetAttributes(&a, ns_rounds_kernel<3>);
  cudaFuncGetAttributes(&a, ns_rounds_kernel<4>);
  cudaFuncGetAttributes(&a, ns_rounds_kernel<6>);
  cudaFuncGetAttributes(&a, ns_rounds_kernel<11>);
}

}  // namespace brawl
