// metropolis_rounds.cu -- Metropolis chains whose lattices the halo and the
// fields do not take (simple cubic; more sites than shared memory holds as bytes)
// in rounds of up to twelve trials: the trials of monte_carlo_step_nbr /
// monte_carlo_step_lattice (src/metropolis.F90:751-891) on the chain's own
// mt19937ar stream, as metropolis_kernel runs them.
//
// Where a trial starts depends on whether those before it went uphill (a word
// more each).  Four warps make the stream and the trial that would start at each
// position (field_engine.cuh's makers).  Twelve warps evaluate a round: the
// positions that the next trials can start at, the nearest first, a position
// each, on the lattice as it is.  The trials are then decided in order, up to one
// whose position was not evaluated or whose sums or sites an accepted one before
// it changed.
//
// The lattice is staged in shared memory, a byte a site or, where that is too
// much, half a byte.
#include "accept_thresholds.cuh"
#include "field_engine.cuh"

namespace brawl {

namespace {

constexpr int kRound = 12;  // positions of a round, one a warp
constexpr int kRoundTeam = 32 * kRound;
constexpr int kRoundMeet = kRoundTeam + 32 * kFieldMakers;
constexpr int kRoundThreads = kRoundMeet;

__device__ __forceinline__ void round_sync() { asm volatile("bar.sync 6, %0;" ::"n"(kRoundTeam) : "memory"); }

// Shared memory of a chain: the stream's rings and the records (FieldLayout's A
// and B), V, the axis tables and F, the entries, the exact tier's terms and the
// lattice.
struct RoundLayout {
  uint32_t I, ents, sstart, vbuf, lat, total;
  uint32_t tab_len[3];
  int32_t F_off;  // (in words from I)
};

__host__ __device__ inline RoundLayout round_layout(const Geom& g, bool nibbles) {
  RoundLayout L;
  const uint32_t nsp = (uint32_t)g.ns + 1;
  L.I = align_up(FieldLayout::kV + (uint32_t)(g.ns * g.ns * g.nsh) * 8, 16);
  L.tab_len[0] = 2 * (uint32_t)g.n1 + 2 * kHalo;
  L.tab_len[1] = 2 * (uint32_t)g.n2 + 2 * kHalo;
  L.tab_len[2] = 2 * (uint32_t)g.n3 + 2 * kHalo;
  L.F_off = (int32_t)(2 * (L.tab_len[0] + L.tab_len[1] + L.tab_len[2]));
  L.ents = L.I + ((uint32_t)L.F_off + nsp * (uint32_t)g.nsh * nsp) * 4;
  L.sstart = L.ents + (uint32_t)g.z * 4;
  L.vbuf = align_up(L.sstart + (uint32_t)(g.nsh + 1) * 2, 16);
  L.lat = align_up(L.vbuf + 4u * (uint32_t)g.z * 8, 16);
  const uint32_t n = (uint32_t)g.n_sites;
  L.total = align_up(L.lat + (nibbles ? (n + 1) / 2 : n), 16);
  return L;
}

// The lattice: a byte a site, or half a byte (the lower half first).
template <bool kNibbles>
struct RoundLat {
  unsigned char* p;
  __device__ __forceinline__ int operator()(int i) const {
    return kNibbles ? (p[i >> 1] >> ((i & 1) << 2)) & 15 : p[i];
  }
  // a site that only this thread writes (its byte's other half may be another's)
  __device__ __forceinline__ void change(int i, int from, int to) const {
    if (kNibbles)
      atomicXor(reinterpret_cast<unsigned*>(p) + (i >> 3), (unsigned)(from ^ to) << ((i & 7) << 2));
    else
      p[i] = (unsigned char)to;
  }
};
static_assert(kMaxSpecies < 16, "species in half a byte");

// What the team shares of a round's positions (twice: one is read while the next
// is written): the change in quanta, and whether an accepted trial changed what it
// was summed from.
struct RoundShare {
  int change[2][kWin];
  int stale[2][kWin];
  int verdict;
};
static_assert(own_bytes<FieldEnd, RoundShare>() == kRoundsOwn, "what the layout leaves room for");

}  // namespace

uint32_t round_smem_bytes(const Geom& g, bool nibbles) { return round_layout(g, nibbles).total; }

// A chain's trials depend on one another, so a round's own chain bounds it: some
// 1,600 cycles, instruction latency for the most part (the positions 480, the
// sums 170 to 500, the decisions 400, the check for what an accepted trial changes
// 200 to 600), for five trials.  metropolis_kernel takes 900 to 1,400 cycles a
// trial, the latencies of its loads one after the other.  4,000 trials: simple
// cubic 6^3, three species, 2.6 ms there and 0.73 ms here; 8^3, two species, 1.65
// and 0.93 (ties, on the exact tier in both); fcc 40^3, four species, from a random
// configuration 2.9 and 0.94.
template <int NJ, bool kNibbles>
__global__ void __launch_bounds__(kRoundThreads, 1) metropolis_rounds_kernel(const ChainJob* __restrict__ jobs) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ FieldEnd end;
  __shared__ __align__(16) RoundShare S;
  const ChainJob& J = jobs[blockIdx.x];
  if (J.status && *J.status != 0) return;  // the chain's input was flagged: no trial runs
  const Geom g = J.g;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned long long t_start = global_ns();
  const RoundLayout L = round_layout(g, kNibbles);
  double* V = reinterpret_cast<double*>(smem + FieldLayout::kV);
  int32_t* I = reinterpret_cast<int32_t*>(smem + L.I);
  uint32_t* ents = reinterpret_cast<uint32_t*>(smem + L.ents);
  int16_t* sstart = reinterpret_cast<int16_t*>(smem + L.sstart);
  const RoundLat<kNibbles> lat{smem + L.lat};
  {
    const int nsp = g.ns + 1;
    for (int i = tid; i < g.ns * g.ns * g.nsh; i += blockDim.x) V[i] = J.V[i];
    for (int i = tid; i < nsp * g.nsh * nsp; i += blockDim.x) I[L.F_off + i] = J.F[i];
    for (int i = tid; i < g.z; i += blockDim.x) ents[i] = J.entries[i];
    for (int i = tid; i <= g.nsh; i += blockDim.x) sstart[i] = J.shell_start[i];
    const int n4 = g.n_sites >> 2;
    const uint32_t* src = reinterpret_cast<const uint32_t*>(J.lat);
    if (kNibbles) {
      for (int i = tid; i < n4; i += blockDim.x) {
        const uint32_t w = src[i], v = w | w >> 4;  // (a byte's upper half is zero)
        reinterpret_cast<uint16_t*>(lat.p)[i] = (uint16_t)((v & 0xffu) | (v >> 8 & 0xff00u));
      }
      for (int i = 2 * n4 + tid; i < (g.n_sites + 1) / 2; i += blockDim.x) {
        const int hi = 2 * i + 1 < g.n_sites ? J.lat[2 * i + 1] : 0;
        lat.p[i] = (unsigned char)(J.lat[2 * i] | hi << 4);
      }
    } else {
      for (int i = tid; i < n4; i += blockDim.x) reinterpret_cast<uint32_t*>(lat.p)[i] = src[i];
      for (int i = 4 * n4 + tid; i < g.n_sites; i += blockDim.x) lat.p[i] = (unsigned char)J.lat[i];
    }
  }
  AxisTables T;
  build_axis_tables(g, I, L.tab_len, lane, T);  // (every warp, the same values)
  if (tid == 0) end.done = 0;
  __syncthreads();
  const bool nbr = J.nbr_swap != 0;
  if (warp < kFieldMakers) {
    // records: A  indices of site 1 and 2; a change above A.z is rejected; the
    //             acceptance word
    //          B  their coordinates; an uphill change below B.z is accepted
    const int band = J.band;
    const float inv_k = 1.0f / J.beta_q_l2, band_f = (float)band;
    stream_produce<kRoundMeet>(J.rng, smem, &end, warp, lane, [&](const uint32_t* w, int slot) {
      int ax, ay, az, bx, by, bz;
      draw_site(g, w[0], w[1], w[2], ax, ay, az);
      if (nbr) draw_nbr(g, w[3], ax, ay, az, bx, by, bz);
      else draw_site(g, w[3], w[4], w[5], bx, by, bz);
      const uint32_t wu = w[nbr ? 4 : 6];
      const AcceptThresholds th = accept_thresholds(wu, inv_k, band_f);
      *reinterpret_cast<int4*>(smem + FieldLayout::kA + slot * 16) = make_int4(
          compact_index(g, ax, ay, az), compact_index(g, bx, by, bz), max(band, th.rej_above), (int)wu);
      *reinterpret_cast<int4*>(smem + FieldLayout::kB + slot * 16) =
          make_int4(ax | ay << 10 | az << 20, bx | by << 10 | bz << 20, th.acc_below, 0);
    });
  } else {
    const int mine = warp - kFieldMakers, tt = mine * 32 + lane;  // the round's trial
    const bool second = lane >= 16;                               // its site 2
    // this lane's entries: every 16th
    int ex[NJ], ey[NJ], ez[NJ], shp[NJ];
    unsigned valid = 0;
    {
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
          valid |= 1u << j;
        }
        ex[j] = at(T.tx[sc && dx == 0], dx);
        ey[j] = at(T.ty[sc && dy == 0], dy);
        ez[j] = at(T.tz[sc && dz == 0], dz);
        shp[j] = 4 * sh * (g.ns + 1);
      }
    }
    double* vbuf = reinterpret_cast<double*>(smem + L.vbuf);
    const int F_at = (int)L.I + 4 * L.F_off, row_bytes = 4 * g.nsh * (g.ns + 1);
    auto word = [&](int at) { return *reinterpret_cast<const int32_t*>(smem + at); };
    const int band = J.band, n_base = nbr ? 4 : 6;
    const int nt = (int)J.n_trials;
    int t = 0;
    unsigned c_eval = 0, c_acc = 0, c_like = 0, c_exact = 0;
    DecideStats stats = {0u, 0u};
    unsigned n_win = 0;  // windows of the stream passed
    int o = 0;           // the next trial's position in the window
    unsigned have = 0;   // the last part waited for
    int flip = 0;        // the results in use
    // k <= 64 words on; the next 32 positions' records are at hand
    auto advance = [&](int k) {
      o += k;
      const unsigned before = n_win / kFieldMakers;
      n_win += (unsigned)(o >> 5);
      o &= kWin - 1;
      if (n_win / kFieldMakers != before) used_arrive<kRoundMeet>((int)(before & 1u));
      if ((n_win + 1) / kFieldMakers != have) {
        ++have;
        made_wait<kRoundMeet>((int)(have & 1u));
      }
    };
    auto rec = [&](uint32_t at, unsigned r) {
      return *reinterpret_cast<const int4*>(smem + at + (r & (kFieldRing - 1)) * 16);
    };
    made_wait<kRoundMeet>(0);
    while (t < nt) {
      // ---- the positions: lane p has the next p-th --------------------------
      const unsigned r0 = n_win * kWin + (unsigned)o;
      const int4 a = rec(FieldLayout::kA, r0 + lane), b = rec(FieldLayout::kB, r0 + lane);
      const int s_a = lat(a.x), s_b = lat(a.y);
      const unsigned like = __ballot_sync(kFull, s_a == s_b);
      // where trials can start: a like pair draws n_base words, another one more
      // when it goes uphill
      unsigned can = 1u, at_level = 1u;
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        at_level = (at_level << n_base) | ((at_level & ~like) << (n_base + 1));
        can |= at_level;
      }
      if (nbr) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          at_level = (at_level << n_base) | ((at_level & ~like) << (n_base + 1));
          can |= at_level;
        }
      }
      // this warp's: the mine-th of the unlike ones
      const unsigned lt = (1u << lane) - 1u;
      const int rank = __popc(can & ~like & lt);
      const bool unlike = (can & ~like) >> lane & 1u;
      const unsigned evaluated = __ballot_sync(kFull, unlike && rank < kRound);
      const unsigned mine_m = __ballot_sync(kFull, unlike && rank == mine);
      const int p = __ffs(mine_m) - 1;
      const int a_at = __shfl_sync(kFull, a.x, p & 31), b_at = __shfl_sync(kFull, a.y, p & 31);
      const int xyz1 = __shfl_sync(kFull, b.x, p & 31), xyz2 = __shfl_sync(kFull, b.y, p & 31);
      const int both = __shfl_sync(kFull, s_a | s_b << 8, p & 31);
      const int sa = both & 0xff, sb = both >> 8;
      const int xyz = second ? xyz2 : xyz1, own = second ? b_at : a_at, other = second ? a_at : b_at;
      const int so = second ? sb : sa, sn = second ? sa : sb;
      int ni[NJ];
      if (p >= 0) {
        const int cx = (xyz & 1023) << 2, cy = (xyz >> 8) & 4092, cz = (xyz >> 18) & 4092;
        const int rowN = F_at + sn * row_bytes, rowO = F_at + so * row_bytes;
        int s[NJ];
#pragma unroll
        for (int j = 0; j < NJ; ++j) ni[j] = word(ex[j] + cx) + word(ey[j] + cy) + word(ez[j] + cz);
#pragma unroll
        for (int j = 0; j < NJ; ++j) s[j] = lat(ni[j]);
        int dE = 0;
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          // after the swap the other site holds our old species
          const int then = ni[j] == other ? so : s[j];
          const int v = word(rowN + shp[j] + 4 * then) - word(rowO + shp[j] + 4 * s[j]);
          dE += (valid >> j) & 1u ? v : 0;
          if (!((valid >> j) & 1u)) ni[j] = -1;
        }
        dE = __reduce_add_sync(kFull, dE);
        if (lane == 0) S.change[flip][p] = dE;
      }
      round_sync();
      // ---- the decisions, in order -------------------------------------------
      const bool known = (evaluated >> lane) & 1u;
      const int d = known ? S.change[flip][lane] : 0;
      const unsigned rej = __ballot_sync(kFull, known && d > a.z);
      const unsigned acc7 = __ballot_sync(kFull, known && d > band && d <= a.z && d < b.z);
      const unsigned acc6 = __ballot_sync(kFull, known && d < -band);
      const unsigned six = like | acc6, seven = rej | acc7;
      unsigned path = 1u;
#pragma unroll
      for (int i = 0; i < 5; ++i) path |= ((path & six) << n_base) | ((path & seven) << (n_base + 1));
      if (nbr) {
#pragma unroll
        for (int i = 0; i < 2; ++i) path |= ((path & six) << n_base) | ((path & seven) << (n_base + 1));
      }
      unsigned trials = path & (six | seven);
      // no more than the run has left
      if (__popc(trials) > nt - t) trials &= __ballot_sync(kFull, __popc(trials & lt) < nt - t);
      // up to a trial that an accepted one before it changes: its sites, or a site
      // that it was summed from
      unsigned took = trials & (acc6 | acc7);
      if (took && (trials >> (__ffs(took) - 1)) > 1u) {
        bool same = false, stale = false;
        // (the last trial of the path has none after it)
        for (unsigned m = took & ~(1u << (31 - __clz(trials))); m; m &= m - 1u) {
          const int k = __ffs(m) - 1;
          const int ca = __shfl_sync(kFull, a.x, k), cb = __shfl_sync(kFull, a.y, k);
          const bool met = (a.x == ca) | (a.x == cb) | (a.y == ca) | (a.y == cb);
          same |= lane > k && met;
          bool hit = false;
#pragma unroll
          for (int j = 0; j < NJ; ++j) hit |= (ni[j] == ca) | (ni[j] == cb);
          stale |= p > k && hit;
        }
        unsigned cut = __ballot_sync(kFull, same);
        stale = __any_sync(kFull, stale);
        if (lane == 0 && p >= 0) S.stale[flip][p] = stale;
        round_sync();
        cut |= __ballot_sync(kFull, known && S.stale[flip][lane] != 0);
        cut &= trials;
        if (cut) trials &= (cut & (0u - cut)) - 1u;
        took &= trials;
      }
      flip ^= 1;
      int next;  // the next trial's position
      if (trials == 0) {
        // inside the band, or too near its threshold: the reference's FP64 sums, in
        // its order
        ++c_exact;
        if (mine == 0) {  // (the first position is the first warp's)
          SitePair q;
          q.ax = xyz1 & 1023;
          q.ay = (xyz1 >> 10) & 1023;
          q.az = xyz1 >> 20;
          q.bx = xyz2 & 1023;
          q.by = (xyz2 >> 10) & 1023;
          q.bz = xyz2 >> 20;
          q.ai = a_at;
          q.bi = b_at;
          q.sa = sa;
          q.sb = sb;
          double e_un, e_sw;
          exact_pair_energies_staged(g, lat, V, ents, sstart, q, lane, e_un, e_sw, vbuf);
          const double delta_e = __dsub_rn(e_sw, e_un);
          int verdict = 1;
          if (!(delta_e < 0.0)) {
            const uint32_t wu = (uint32_t)__shfl_sync(kFull, a.w, 0);
            verdict = u_lt_exp(wu, __dmul_rn(-J.beta, delta_e), stats) | 2;
          }
          if (lane == 0) S.verdict = verdict;
        }
        round_sync();
        const int verdict = *(volatile int*)&S.verdict;
        took = verdict & 1;
        trials = 1u;
        next = n_base + (verdict >> 1);
      } else {
        const int last = 31 - __clz(trials);
        next = last + n_base + (int)((seven >> last) & 1u);
      }
      if (p >= 0 && (took >> p) & 1u && (lane & 15) == 0) lat.change(own, so, sn);
      t += __popc(trials);
      c_like += __popc(trials & like);
      c_eval += __popc(trials & ~like);
      c_acc += __popc(took);
      advance(next);
      if (took) round_sync();
    }
    const unsigned long long drawn = (unsigned long long)kWin * n_win + (unsigned long long)o;
    // the makers have made, or are making, the part after this one and then wait
    // for this one to be used
    const unsigned part = n_win / kFieldMakers;
    if (have == part) made_wait<kRoundMeet>((int)((part + 1) & 1u));
    if (tt == 0) {
      end.words = drawn;
      end.done = 1;
    }
    __syncwarp();
    used_arrive<kRoundMeet>((int)(part & 1u));
    if (tt == 0) {
      unsigned long long* c = J.counters;
      c[kCntTrials] += (unsigned long long)nt;
      c[kCntEvaluated] += c_eval;
      c[kCntDraws] += drawn;
      c[kCntAccepted] += (unsigned long long)c_like + c_acc;
      c[kCntExpTests] += drawn - (unsigned long long)n_base * (unsigned long long)nt;
      c[kCntExactPath] += c_exact;
      c[kCntExpFp64] += stats.fp64;
      c[kCntExpCr] += stats.cr;
    }
  }
  __syncthreads();
  // ---- write back -----------------------------------------------------------
  {
    const int n4 = g.n_sites >> 2;
    uint32_t* dst = reinterpret_cast<uint32_t*>(J.lat);
    if (kNibbles) {
      for (int i = tid; i < n4; i += blockDim.x) {
        const uint32_t h = reinterpret_cast<const uint16_t*>(lat.p)[i], v = (h & 0xffu) | (h & 0xff00u) << 8;
        dst[i] = (v & 0x000f000fu) | (v & 0x00f000f0u) << 4;
      }
    } else {
      for (int i = tid; i < n4; i += blockDim.x) dst[i] = reinterpret_cast<const uint32_t*>(lat.p)[i];
    }
    for (int i = 4 * n4 + tid; i < g.n_sites; i += blockDim.x) J.lat[i] = (int8_t)lat(i);
  }
  if (tid == 0 && J.t_ns) *J.t_ns = global_ns() - t_start;
}

template <int NJ, bool kNibbles>
static void launch_rounds_lat(const ChainJob* d_jobs, int n_jobs, uint32_t smem_bytes, cudaStream_t stream) {
  BRAWL_SHARED(kRoundsOwn, (metropolis_rounds_kernel<NJ, kNibbles>));
  metropolis_rounds_kernel<NJ, kNibbles><<<n_jobs, kRoundThreads, smem_bytes, stream>>>(d_jobs);
}

template <int NJ>
static void launch_rounds_nj(const ChainJob* d_jobs, int n_jobs, bool nibbles, uint32_t smem_bytes,
                             cudaStream_t stream) {
  if (nibbles) launch_rounds_lat<NJ, true>(d_jobs, n_jobs, smem_bytes, stream);
  else launch_rounds_lat<NJ, false>(d_jobs, n_jobs, smem_bytes, stream);
}

void launch_metropolis_rounds(const ChainJob* d_jobs, int n_jobs, bool nibbles, uint32_t smem_bytes, int max_z,
                              cudaStream_t stream) {
  if (n_jobs <= 0) return;
  if (max_z <= 32) launch_rounds_nj<2>(d_jobs, n_jobs, nibbles, smem_bytes, stream);
  else if (max_z <= 64) launch_rounds_nj<4>(d_jobs, n_jobs, nibbles, smem_bytes, stream);
  else if (max_z <= 96) launch_rounds_nj<6>(d_jobs, n_jobs, nibbles, smem_bytes, stream);
  else launch_rounds_nj<11>(d_jobs, n_jobs, nibbles, smem_bytes, stream);
}

}  // namespace brawl
