// metropolis_halo.cu -- Metropolis-Kawasaki swap trials for fcc/bcc chains
// staged with a periodic halo (see halo_shear.cuh): the batched path's
// kernel for every lattice that fits.  One warp (CTA) per chain; trials in
// the reference's order (monte_carlo_step_lattice / _nbr,
// src/metropolis.F90:751-891) on the chain's own mt19937ar stream.

#include "accept_thresholds.cuh"
#include "halo_engine.cuh"
#include "halo_shear.cuh"
#include "kernels.cuh"

namespace brawl {

// A stream position's record: the trial that would start there.
//   rec    (cell of site 1, row of site 1, cell of site 2, row of site 2): the
//          cell in the sheared lattice, the row of the difference table (byte
//          address) for the site's species changing to the other site's
//   flags  bits 0-5, 6-11: 4 times the species of site 1, site 2; bit 12: the
//          pair may be within interaction range; bits 13-16: the neighbour
//          drawn (nearest-neighbour swaps); bits 17-22, 23-28: per axis (x, y,
//          z) of site 1, site 2 whether it has an image one period up (1) or
//          down (2)
constexpr int kFlagNear = 1 << 12, kFlagNbr = 13, kFlagImg1 = 17, kFlagImg2 = 23;
constexpr int kFlagSpecies = (1 << 12) - 1;

// The reference-order FP64 decision (see metropolis.cu) of a trial: bit 0
// accept, bit 1 uniform drawn, bit 2 FP64 libm tier, bit 3 double-double.
// Lane c < 4 nsh adds, in list order from 0.0, the terms of shell c % nsh of
// evaluation c / nsh (site 1 before, site 2 before, site 1 after, site 2
// after); the shell sums are then added in shell order and the two sites'
// energies summed (nbr_energy and pair_energy,
// src/bw_hamiltonian.f90:99-114).  After the swap an entry whose neighbour is
// the other site (its displacement is the pair's, d; -2 for a pair that is not
// near) finds our old species there.  Each chain's loop is unrolled by four,
// so the loads of four terms issue ahead of their adds.
static __device__ __noinline__ int window_exact(const ChainJob* __restrict__ Jg, const double* V,
                                                const int32_t* edelta, const int32_t* ecan, int epad,
                                                const int16_t* sstart, const uint8_t* lat, int ca, int cb, int sa,
                                                int sb, int d, int ns, int nsh, uint32_t wu, int lane) {
  const int nc = 4 * nsh;
  double part[2] = {0.0, 0.0};
#pragma unroll 1
  for (int r = 0; r < 2; ++r) {
    const int c = lane + 32 * r;
    double sum = 0.0;
    if (c < nc) {
      const int ev = c / nsh, sh = c - ev * nsh;
      const bool on2 = ev & 1, after = ev >= 2;
      const uint8_t* at = lat + (on2 ? cb : ca);
      const int own = on2 ? sb : sa, other = on2 ? sa : sb;
      const int cs = after ? other : own;
      // Vr[ns * s] = V(cs, s, sh) for the neighbour species s (1-based)
      const double* Vr = V + (cs - 1) + ns * ns * sh - ns;
      const int k1 = sstart[sh + 1];
      if (d != -2 && after) {
        const int32_t* E = ecan + (on2 ? epad : 0);
        for (int k = sstart[sh]; k < k1; ++k)
          sum = __dadd_rn(sum, Vr[ns * (E[k] == d ? own : (int)at[edelta[k]] >> 2)]);
      } else {
#pragma unroll 4
        for (int k = sstart[sh]; k < k1; ++k) sum = __dadd_rn(sum, Vr[ns * ((int)at[edelta[k]] >> 2)]);
      }
    }
    part[r] = sum;
  }
  double e_un, e_sw;
  combine_pair_energies(part, nsh, lane, e_un, e_sw);
  const double delta_e = __dsub_rn(e_sw, e_un);
  if (delta_e < 0.0) return 1;
  DecideStats st = {0u, 0u};
  const int acc = u_lt_exp(wu, __dmul_rn(-Jg->beta, delta_e), st);
  return acc | 2 | (st.fp64 ? 4 : 0) | (st.cr ? 8 : 0);
}

// site_2 - site_1 modulo the periods, one number (the entries' ecan values).
__device__ __forceinline__ int displacement(const Geom& g, int dx, int dy, int dz) {
  const int W1 = 2 * g.n1, W2 = 2 * g.n2, W3 = 2 * g.n3;
  return (dx < 0 ? dx + W1 : dx) + W1 * ((dy < 0 ? dy + W2 : dy) + W2 * (dz < 0 ? dz + W3 : dz));
}

__device__ __forceinline__ int image_codes(const HaloGeom& H, int X, int Y, int Z) {
  const int cx = X < H.hx ? 1 : (X >= H.NX - H.hx ? 2 : 0);
  const int cy = Y < H.hy ? 4 : (Y >= H.NY - H.hy ? 8 : 0);
  const int cz = Z < H.hz ? 16 : (Z >= H.NZ - H.hz ? 32 : 0);
  return cx | cy | cz;
}

constexpr int kNoTrial = 0x40;  // no further trial known: past the two windows, or too many like pairs between
constexpr int kRun = 5;         // like pairs a step passes over at most, plus one

// Where the next kSpec trials of unlike species start from position o of the
// first window if each of them draws its uniform, one byte each, kNoTrial when
// not known.  lo, hi: the two windows' masks of unlike pairs; every: the
// positions a run of like pairs steps through, n_base apart (bits 0, n_base,
// ..., 4 n_base).
template <int kSpec>
__device__ __forceinline__ unsigned win_chain(unsigned lo, unsigned hi, int o, int n_base, unsigned every) {
  unsigned pos = 0;
  unsigned a = __funnelshift_r(lo, hi, o), b = hi >> o;
  bool known = true;
#pragma unroll
  for (int k = 0; k < kSpec; ++k) {
    const unsigned m = a & every;
    const int s = __ffs(m) - 1;
    known = known && m != 0u;
    pos |= (unsigned)(known ? o + s : kNoTrial) << (8 * k);
    const int step = s + n_base + 1;  // at most 31
    o += step;
    a = __funnelshift_r(a, b, step);
    b >>= step;
  }
  return pos;
}

// One warp per chain.  What bounds it: a chain's trials are one dependent
// sequence, so the instructions and latencies of a trial times the longest
// chain's trials are the launch's time; shared-memory bandwidth is far from
// its limit.  Two things shorten the sequence.
//
// What the stream alone decides -- sites, cells, which pairs are unlike -- is
// decoded for 32 stream positions at once, one per lane (trial_window.cuh),
// into records in shared memory.
//
// kSpec trials are evaluated together.  Most evaluated trials go uphill and are
// rejected (87% at 900 K on bcc with four species, 70% at 3000 K): they leave
// the lattice as it is and draw their uniform, so the next trial starts seven
// words on.  The batch takes the next kSpec trials on that assumption; their
// loads, sums and tests overlap, and the trials up to and including the first
// that is not a certain rejection are the chain's trials, in order, on the
// lattice they would have seen.  The rest are dropped and drawn again from where
// the stream then stands.
//
// Very hot chains accept most trials, and take one at a time (gather_trials).
// Every lane then has the trial's record and its change, so no vote is needed, and
// what an accepted swap writes is made ready beside the sums.  400 chains of bcc
// 14^3, five species, two shells, 4,000 trials: 1.46 ms at 4000 K and 1.58 at
// infinite temperature; as rounds of one with the votes of the longer ones 1.71 and
// 1.93, and 1.62 and 1.65 without windows, trial by trial.
template <int NJ, int kSpec>
// (16 blocks an SM: without a bound the compiler spills the rounds of one, and the
// short lists lose 3%)
__global__ void __launch_bounds__(32, kSpec == 1 || NJ == 2 ? 16 : 0) metropolis_halo_kernel(const ChainJob* __restrict__ jobs) {
  extern __shared__ __align__(16) unsigned char smem[];
  using WL = WindowLayout;
  const ChainJob* Jg = jobs + blockIdx.x;
  if (Jg->status && *Jg->status != 0) return;  // the chain's input was flagged: no trial runs
  const Geom g = Jg->g;
  const HaloGeom H = Jg->hg;
  const int lane = threadIdx.x;
  __shared__ unsigned long long s_t_start;  // kept out of registers
  if (lane == 0) s_t_start = global_ns();
  const WindowLayout L = window_layout(g, H);
  uint32_t* mt = reinterpret_cast<uint32_t*>(smem);
  uint32_t* tw = mt + GatherRing::kTwAt;
  int4* rec = reinterpret_cast<int4*>(smem + WL::kRec);
  int32_t* flags = reinterpret_cast<int32_t*>(smem + WL::kFlags);
  uint8_t* lat = smem + WL::kLat;
  double* V = reinterpret_cast<double*>(smem + L.V);
  int32_t* F = reinterpret_cast<int32_t*>(smem + L.I);
  int32_t* edelta = reinterpret_cast<int32_t*>(smem + L.edelta);
  int32_t* ecan = reinterpret_cast<int32_t*>(smem + L.ecan);
  int32_t* dnbr = reinterpret_cast<int32_t*>(smem + L.dnbr);
  int16_t* sstart = reinterpret_cast<int16_t*>(smem + L.sstart);
  const bool bcc = g.lattice == kBcc;
  const bool nbr_swap = Jg->nbr_swap != 0;
  const int nsp = g.ns + 1;
  const int epad = entry_pad(g.z);

  // ---- stage state ------------------------------------------------------
  const int nF = nsp * g.nsh * nsp, nV = g.ns * g.ns * g.nsh;
  const uint32_t* rng = Jg->rng;
  const int pos0 = (int)rng[kMTN];
  mt_roll_load<GatherRing>(rng, mt, pos0, lane);
  for (int i = lane; i < nF; i += 32) F[i] = Jg->F[i];
  {
    // the difference table, each pair's rows followed by a row of zeros (for
    // the lane entries past z)
    int32_t* D = reinterpret_cast<int32_t*>(smem + L.D);
    const int per = g.nsh * nsp, all = L.Dk / 4;
#pragma unroll 4
    for (int i = lane; i < nsp * nsp * all; i += 32) {
      const int p = i / all, r = i - p * all;
      D[i] = r < per ? Jg->F[nF + p * per + r] : 0;
    }
  }
  for (int i = lane; i < nV; i += 32) V[i] = Jg->V[i];
  for (int i = lane; i <= g.nsh; i += 32) sstart[i] = Jg->shell_start[i];
  for (int k = lane; k < epad; k += 32) {
    int e1 = -1, e2 = -1;  // no entry: matches no displacement
    if (k < g.z) {
      int dx, dy, dz, sh;
      unpack_entry(Jg->entries[k], dx, dy, dz, sh);
      edelta[k] = shear_step(bcc, H, dx, dy, dz);
      // the displacement site 2 - site 1 that makes the entry's neighbour of
      // site 1, of site 2, the other site
      e1 = displacement(g, dx, dy, dz);
      e2 = displacement(g, -dx, -dy, -dz);
    }
    ecan[k] = e1;
    ecan[epad + k] = e2;
  }
  if (lane < g.nbr_k) {
    const int8_t* v = cNbrSwap[g.lattice][lane];
    dnbr[lane] = displacement(g, v[0], v[1], v[2]);
  }
  shear_fill(g, H, Jg->lat, lat, lane);
  __syncwarp();
  // lanes 0-15 sum site 1's neighbours, 16-31 site 2's; lane l the entries
  // (l & 15) + 16 j, the ones past z on the zero row
  const bool on_b = lane >= 16;
  int step[NJ], shp[NJ];
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const int k = (lane & 15) + 16 * j;
    step[j] = k < g.z ? edelta[k] : 0;
    shp[j] = (k < g.z ? (int)(Jg->entries[k] >> 24) : g.nsh) * nsp * 4;
  }
  const int band = Jg->band;
  const float inv_k = 1.0f / Jg->beta_q_l2, band_f = (float)band;
  const int n_base = nbr_swap ? 4 : 6;
  const unsigned every = nbr_swap ? 0x00011111u : 0x01041041u;
  const unsigned inv_base = nbr_swap ? 64u : 43u;  // i inv_base >> 8 = i / n_base for multiples i < 80
  const int nt = (int)Jg->n_trials;
  const int Dk = L.Dk, D_at = (int)L.D;
  const int img_axes = ((lane & 1) ? 3 : 0) | ((lane & 2) ? 12 : 0) | ((lane & 4) ? 48 : 0);
  const int img_at = lane < 8 ? kFlagImg1 : kFlagImg2;
  // 32-bit tallies (a launch runs fewer than 2^31 trials per chain, see
  // launch_metropolis_halo); the uniforms follow from the words consumed
  unsigned int b_eval = 0, b_acc = 0, b_exact = 0;
  unsigned int c_fp64 = 0, c_cr = 0;

  // ---- the stream -----------------------------------------------------------
  MtRoll R = {pos0, 0, 0};
#pragma unroll 1
  for (int i = 0; i < kLookAhead / kWin; ++i) {
    mt_roll<GatherRing>(mt, tw, R, lane);
    __syncwarp();
  }
  unsigned int n_win = 0;   // windows passed
  int tb = GatherRing::kTw - 2 * kWin;  // the first window's place in the ring of tempered words
  int half = 0;             // its half of the record ring: 0 or kWin
  // this lane's sites: of the two windows, and of the next one (species not
  // read yet, the pair's flags in nf)
  int ca0, cb0, ca1 = 0, cb1 = 0, na, nb, nf;
  unsigned lo = 0, hi = 0;  // the windows' masks of unlike pairs
  auto decode = [&](int at) {
    const uint32_t* w = tw + at + lane;
    int x, y, z, Y, X, x2, y2, z2, Y2, X2;
    draw_site_halo(g, bcc, w[0], w[1], w[2], x, y, z, Y, X);
    if (!nbr_swap) {
      draw_site_halo(g, bcc, w[3], w[4], w[5], x2, y2, z2, Y2, X2);
      nf = words_near(H.near_c, H.near_2c, w) ? kFlagNear : 0;
    } else {
      // draw_nbr's neighbour; its steps are -1, 0, 1
      const int k = (int)umulhi32(w[3], (uint32_t)g.nbr_k);
      const int8_t* v = cNbrSwap[g.lattice][k];
      x2 = wrap_fast(x + v[0], 2 * g.n1);
      y2 = wrap_fast(y + v[1], 2 * g.n2);
      z2 = wrap_fast(z + v[2], 2 * g.n3);
      Y2 = y2 >> g.ys;
      X2 = x2 >> 1;
      nf = kFlagNear | k << kFlagNbr;
    }
    na = shear_cell(bcc, H, z, Y, X);
    nb = shear_cell(bcc, H, z2, Y2, X2);
    nf |= image_codes(H, X, Y, z) << kFlagImg1 | image_codes(H, X2, Y2, z2) << kFlagImg2;
  };
  auto put = [&](int slot, int ca, int cb, int sa4, int sb4, int f) {
    // rows of the species pairs: D + (so (ns + 1) + sn) Dk
    const int ra = D_at + ((sa4 * nsp + sb4) >> 2) * Dk, rb = D_at + ((sb4 * nsp + sa4) >> 2) * Dk;
    rec[slot] = make_int4(ca, ra, cb, rb);
    flags[slot] = f | sa4 | sb4 << 6;
  };
  decode(0);
  // one window on: the second becomes the first, the next one's species are
  // read, the one after is decoded and 32 more words are generated
  auto advance = [&]() {
    tb = tb + kWin == GatherRing::kTw ? 0 : tb + kWin;
    ca0 = ca1;
    cb0 = cb1;
    lo = hi;
    ca1 = na;
    cb1 = nb;
    const int f = nf;
    const int sa = lat[na], sb = lat[nb];
    const int ahead = tb + 2 * kWin;
    decode(ahead >= GatherRing::kTw ? ahead - GatherRing::kTw : ahead);
    mt_roll<GatherRing>(mt, tw, R, lane);
    put(half + lane, ca1, cb1, sa, sb, f);  // the half the window that ended held
    half ^= kWin;
    hi = __ballot_sync(kFull, sa != sb);
    __syncwarp();
  };
  advance();
  advance();
  int o = 0;  // the next trial's position in the first window
  int t = 0;

  while (t < nt) {
    while (o >= kWin) {
      o -= kWin;
      advance();
      ++n_win;
    }
    const unsigned pos = win_chain<kSpec>(lo, hi, o, n_base, every);
    int n_known = kSpec;  // the trials of the batch that are known to follow
    if (nt - t < kWin) {
      // the run ends here or soon: one trial at a time
      const int like = (pos & kNoTrial) ? kRun : (int)(((unsigned)((int)(pos & 0xff) - o) * inv_base) >> 8);
      if ((pos & kNoTrial) || like >= nt - t) {
        const int m = min(nt - t, like);
        t += m;
        b_acc += m;
        o += m * n_base;
        continue;
      }
      n_known = 1;
    } else if (pos & kNoTrial) {
      // a run of like pairs: accepted without an energy evaluation or a draw
      t += kRun;
      b_acc += kRun;
      o += kRun * n_base;
      continue;
    }
    // ---- the batch's energy changes ---------------------------------------
    // this lane's word of the batch: trial (lane & 3)'s
    const int pl = (int)((pos >> (8 * min(lane & 3, kSpec - 1))) & 0xff);
    int2 v[kSpec];
    int4 q{};  // the record of the trial that ends the batch: with one, its own
    if constexpr (kSpec == 1) {
      q = rec[(half + pl) & (kRecRing - 1)];
      v[0] = on_b ? make_int2(q.z, q.w) : make_int2(q.x, q.y);
    } else {
#pragma unroll
      for (int k = 0; k < kSpec; ++k) {
        const int slot = (half + (int)((pos >> (8 * k)) & 0xff)) & (kRecRing - 1);
        v[k] = *reinterpret_cast<const int2*>(smem + WL::kRec + slot * 16 + (on_b ? 8 : 0));
      }
    }
    const int fl = flags[(half + pl) & (kRecRing - 1)];
    int wat = tb + pl + n_base;
    wat -= wat >= GatherRing::kTw ? GatherRing::kTw : 0;
    const AcceptThresholds th = accept_thresholds(tw[wat], inv_k, band_f);
    // What a swap of the sites of record q at position p writes: this lane's cell
    // (-1: none), and whether records of the two windows, of the positions still to
    // come, name either site.  (Of one trial it is at hand when the sum is.)
    int cell;
    bool renews;
    auto touched = [&](int p, int f) {
      // the cells of the swapped sites: lanes 0-7 site 1's, 8-15 site 2's; lane
      // c of eight shifts by a period along the axes that its bits name
      const int code = (f >> img_at) & img_axes;
      cell = lane < 8 ? q.x : q.z;
      cell += (code & 1) ? H.kx : ((code & 2) ? -H.kx : 0);
      cell += (code & 4) ? H.ky : ((code & 8) ? -H.ky : 0);
      cell += (code & 16) ? H.kz : ((code & 32) ? -H.kz : 0);
      // every axis of this lane has an image there
      cell = (lane >= 16) | (((code | code >> 1) & 0x15) != (img_axes & 0x15)) ? -1 : cell;
      const bool in0 = (ca0 == q.x) | (ca0 == q.z) | (cb0 == q.x) | (cb0 == q.z);
      const bool in1 = (ca1 == q.x) | (ca1 == q.z) | (cb1 == q.x) | (cb1 == q.z);
      renews = __any_sync(kFull, ((lane > p) & in0) | ((kWin + lane > p) & in1));
    };
    if constexpr (kSpec == 1) touched(pl, fl);
    int acc[kSpec];
#pragma unroll
    for (int k = 0; k < kSpec; ++k) acc[k] = 0;
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      int s[kSpec];
#pragma unroll
      for (int k = 0; k < kSpec; ++k) s[k] = smem[WL::kLat + (unsigned)(v[k].x + step[j])];
#pragma unroll
      for (int k = 0; k < kSpec; ++k)
        acc[k] += *reinterpret_cast<const int32_t*>(smem + (unsigned)(v[k].y + shp[j] + s[k]));
    }
    unsigned near;
    if constexpr (kSpec == 1) near = (fl & kFlagNear) ? 1u : 0u;
    else near = __ballot_sync(kFull, (fl & kFlagNear) != 0) & ((1u << kSpec) - 1u);
    auto pair_d = [&](int p, int f) {
      // the displacement of the pair at position p
      if (nbr_swap) return dnbr[(f >> kFlagNbr) & 15];
      int ax, ay, az, bx, by, bz;
      const uint32_t* w = tw + (tb + p >= GatherRing::kTw ? tb + p - GatherRing::kTw : tb + p);
      draw_site(g, w[0], w[1], w[2], ax, ay, az);
      draw_site(g, w[3], w[4], w[5], bx, by, bz);
      return displacement(g, bx - ax, by - ay, bz - az);
    };
    if (near) {
      // an entry whose neighbour is the other site: that site holds our old
      // species after the swap, not its own
      const int32_t* E = ecan + (on_b ? epad : 0) + (lane & 15);
      // trial (lane & 3)'s displacement; two sites apart match no entry
      const int dl = pair_d(pl & (kNoTrial - 1), fl);
#pragma unroll
      for (int k = 0; k < kSpec; ++k)
        if ((near >> k) & 1u) {
          const int d = kSpec == 1 ? dl : __shfl_sync(kFull, dl, k), f = kSpec == 1 ? fl : __shfl_sync(kFull, fl, k);
          const int s1 = f & 63, s2 = (f >> 6) & 63;
          const int so = on_b ? s2 : s1, sn = on_b ? s1 : s2;
          const unsigned char* rowN = smem + L.I + (sn >> 2) * g.nsh * nsp * 4;
#pragma unroll
          for (int j = 0; j < NJ; ++j)
            if (16 * j < epad && E[16 * j] == d)
              acc[k] += *reinterpret_cast<const int32_t*>(rowN + shp[j] + so) -
                        *reinterpret_cast<const int32_t*>(rowN + shp[j] + sn);
        }
    }
    // ---- the first trial that is not certainly rejected ---------------------
    // (rej_above >= acc_below: a trial above rej_above is not also below it)
    int p, f;
    bool down, sure;  // its change is below the band; it is accepted
    if constexpr (kSpec == 1) {
      // every lane has the one trial
      const int dE = __reduce_add_sync(kFull, acc[0]);
      down = dE < -band;
      sure = down || (dE > band && dE < th.acc_below);
      p = pl;
      f = fl;
      const int like = (int)(((unsigned)(p - o) * inv_base) >> 8);
      t += like + 1;
      ++b_eval;
      b_acc += like;
      o = p + n_base + 1;
      if (dE > max(band, th.rej_above)) continue;
    } else {
      int dE = 0;  // trial k's in lane k
#pragma unroll
      for (int k = 0; k < kSpec; ++k) {
        const int d = __reduce_add_sync(kFull, acc[k]);
        dE = lane == k ? d : dE;
      }
      const bool mine = lane < n_known && !(pl & kNoTrial);
      const bool below = dE < -band;
      const bool rejected = dE > max(band, th.rej_above);
      const unsigned live = __ballot_sync(kFull, mine);
      const unsigned stop = __ballot_sync(kFull, mine && !rejected);
      const unsigned acc_m = __ballot_sync(kFull, below || (dE > band && dE < th.acc_below));
      const unsigned down_m = __ballot_sync(kFull, below);
      const int last = stop ? __ffs(stop) - 1 : 31 - __clz(live);  // the batch's last trial that counts
      p = (int)((pos >> (8 * last)) & 0xff);
      // trials done: the words passed, less the uniforms, by n_base
      const int done = (int)(((unsigned)(p - o - last) * inv_base) >> 8) + 1;
      t += done;
      b_eval += last + 1;
      b_acc += done - (last + 1);
      o = p + n_base + 1;
      if (stop == 0u) continue;
      const int slot = (half + p) & (kRecRing - 1);
      q = rec[slot];
      f = flags[slot];
      sure = (acc_m >> last) & 1u;
      down = (down_m >> last) & 1u;
    }
    const int s1 = f & 63, s2 = (f >> 6) & 63;
    int accept = 1;
    if (sure) {
      o -= down;
    } else {
      ++b_exact;
      const int d = (f & kFlagNear) ? pair_d(p, f) : -2;
      const int at = tb + p >= GatherRing::kTw ? tb + p - GatherRing::kTw : tb + p;
      const int r = window_exact(Jg, V, edelta, ecan, epad, sstart, lat, q.x, q.z, s1 >> 2, s2 >> 2, d, g.ns, g.nsh,
                                 tw[at + n_base], lane);
      accept = r & 1;
      o -= (r & 2) ? 0 : 1;
      c_fp64 += (r >> 2) & 1;
      c_cr += (r >> 3) & 1;
    }
    if (accept) {
      ++b_acc;
      if constexpr (kSpec > 1) touched(p, f);
      if (cell >= 0) lat[cell] = (uint8_t)(lane < 8 ? s2 : s1);
      if (renews) {
        auto renew = [&](int at, int ca, int cb, bool on) {
          const bool ha = on & ((ca == q.x) | (ca == q.z)), hb = on & ((cb == q.x) | (cb == q.z));
          const int old = flags[at];
          int sa = old & 63, sb = (old >> 6) & 63;
          sa ^= ha ? s1 ^ s2 : 0;
          sb ^= hb ? s1 ^ s2 : 0;
          if (ha | hb) put(at, ca, cb, sa, sb, old & ~kFlagSpecies);
          return sa != sb;
        };
        const bool d0 = renew(half + lane, ca0, cb0, lane > p);
        const bool d1 = renew((half ^ kWin) + lane, ca1, cb1, kWin + lane > p);
        lo = __ballot_sync(kFull, d0);
        hi = __ballot_sync(kFull, d1);
      }
      __syncwarp();  // cells and records are read by the next trials' lanes
    }
  }

  // ---- write back ---------------------------------------------------------
  __syncwarp();
  const unsigned long long words = (unsigned long long)kWin * n_win + (unsigned long long)o;
  shear_store(g, H, lat, Jg->lat, lane);
  mt_roll_store<GatherRing>(mt, tw, R, pos0, words, (unsigned long long)kWin * (n_win + 2) + kLookAhead, Jg->rng, lane);
  if (lane == 0) {
    unsigned long long* c = Jg->counters;
    c[kCntTrials] += (unsigned long long)nt;
    c[kCntEvaluated] += b_eval;
    c[kCntDraws] += words;
    c[kCntAccepted] += b_acc;
    c[kCntExpTests] += words - (unsigned long long)n_base * (unsigned long long)nt;
    c[kCntExactPath] += b_exact;
    c[kCntExpFp64] += c_fp64;
    c[kCntExpCr] += c_cr;
    if (Jg->t_ns) *Jg->t_ns = global_ns() - s_t_start;
  }
}

template <int NJ, int K>
static void launch_halo_nj(const ChainJob* d_jobs, int n_jobs, uint32_t smem_bytes, cudaStream_t stream) {
  BRAWL_SHARED(kOneWarpOwn, metropolis_halo_kernel<NJ, K>);
  metropolis_halo_kernel<NJ, K><<<n_jobs, 32, smem_bytes, stream>>>(d_jobs);
}

template <int NJ>
static void launch_halo_depth(const ChainJob* d_jobs, int n_jobs, uint32_t smem_bytes, int depth, cudaStream_t stream) {
  switch (depth) {
    case 1: launch_halo_nj<NJ, 1>(d_jobs, n_jobs, smem_bytes, stream); break;
    case 2: launch_halo_nj<NJ, 2>(d_jobs, n_jobs, smem_bytes, stream); break;
    case 4: launch_halo_nj<NJ, 4>(d_jobs, n_jobs, smem_bytes, stream); break;
    default: launch_halo_nj<NJ, kGatherDefault>(d_jobs, n_jobs, smem_bytes, stream); break;
  }
}

void launch_metropolis_halo(const ChainJob* d_jobs, int n_jobs, uint32_t smem_bytes, int max_z, int depth,
                            cudaStream_t stream) {
  if (n_jobs <= 0) return;
  switch (lane_entries_for(max_z)) {
    case 2: launch_halo_depth<2>(d_jobs, n_jobs, smem_bytes, depth, stream); break;
    case 4: launch_halo_depth<4>(d_jobs, n_jobs, smem_bytes, depth, stream); break;
    case 6: launch_halo_depth<6>(d_jobs, n_jobs, smem_bytes, depth, stream); break;
    case 8: launch_halo_depth<8>(d_jobs, n_jobs, smem_bytes, depth, stream); break;
    default: launch_halo_depth<11>(d_jobs, n_jobs, smem_bytes, depth, stream); break;
  }
}

template <int K>
static void preload_halo_depth() {
  cudaFuncAttributes a;
  cudaFuncGetAttributes(&a, metropolis_halo_kernel<2, K>);
  cudaFuncGetAttributes(&a, metropolis_halo_kernel<4, K>);
  cudaFuncGetAttributes(&a, metropolis_halo_kernel<6, K>);
  cudaFuncGetAttributes(&a, metropolis_halo_kernel<8, K>);
  cudaFuncGetAttributes(&a, metropolis_halo_kernel<11, K>);
}

// The depths that a server runs chains at.
void preload_halo_kernels() {
  preload_halo_depth<1>();
  preload_halo_depth<kGatherDefault>();
}

}  // namespace brawl
