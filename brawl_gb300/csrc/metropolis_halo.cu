// metropolis_halo.cu -- Metropolis-Kawasaki swap trials for fcc/bcc chains
// staged with a periodic halo (see halo_engine.cuh): the batched path's
// kernel for every lattice that fits.  One warp (CTA) per chain; trials in
// the reference's order (monte_carlo_step_lattice / _nbr,
// src/metropolis.F90:751-891) on the chain's own mt19937ar stream.
#include <climits>

#include "halo_engine.cuh"
#include "kernels.cuh"

namespace brawl {

// Species of canonical compact site i through the halo layout.
struct HaloLat {
  int sz, sy, origin, SZ, SY, off;
  __device__ __forceinline__ int operator()(int i) const {
    extern __shared__ int8_t s_i8[];
    const int Z = i / sz, r = i - Z * sz, Y = r / sy, X = r - Y * sy;
    return s_i8[off + origin + Z * SZ + Y * SY + X];
  }
};

// The reference-order FP64 decision (see metropolis.cu); returns bit 0
// accept, bit 1 uniform drawn, bit 2 FP64 libm tier, bit 3 double-double.
__device__ __noinline__ int halo_exact_decision(const ChainJob* __restrict__ Jg, HaloLat lat,
                                                const double* V, const uint32_t* ents,
                                                const int16_t* sstart, int ax, int ay, int az,
                                                int ai, int bx, int by, int bz, int bi, int sa,
                                                int sb, int lane, uint32_t wu) {
  const Geom g = Jg->g;
  SitePair p;
  p.ax = ax; p.ay = ay; p.az = az; p.ai = ai;
  p.bx = bx; p.by = by; p.bz = bz; p.bi = bi;
  p.sa = sa; p.sb = sb;
  double e_un, e_sw;
  exact_pair_energies(g, lat, V, ents, sstart, p, lane, e_un, e_sw);
  const double delta_e = __dsub_rn(e_sw, e_un);
  if (delta_e < 0.0) return 1;
  DecideStats st = {0u, 0u};
  const int acc = u_lt_exp(wu, __dmul_rn(-Jg->beta, delta_e), st);
  return acc | 2 | (st.fp64 ? 4 : 0) | (st.cr ? 8 : 0);
}

// The species of the neighbour at entry e of a site at padded index `base`
// (relative to the staged lattice) with parity par, through the halo's
// padded offsets (the plan's arithmetic, for any entry).
__device__ __forceinline__ int halo_nbr_species(uint32_t e, int base, int par, int SZ, int SY, bool bcc) {
  extern __shared__ int8_t s_i8[];
  int dx, dy, dz, sh;
  unpack_entry(e, dx, dy, dz, sh);
  const int ddx = (par + dx) >> 1;
  const int ddy = bcc ? ((par + dy) >> 1) : dy;
  return s_i8[base + dz * SZ + ddy * SY + ddx];
}

// halo_exact_decision for a pair that is not near (the pairs halo_delta
// takes): no neighbour of either site is the other, so every neighbour
// holds the same species before and after the swap and is read through
// the padded offsets.  Lane c < 4 nsh adds, in list order from 0.0, the
// terms of shell c % nsh of evaluation c / nsh (site 1 before, site 2
// before, site 1 after, site 2 after); the shell sums are then added in
// shell order and the two sites' energies summed (nbr_energy and
// pair_energy, src/bw_hamiltonian.f90:99-114) -- the values and order of
// exact_pair_energies, so the same doubles.  Each chain's loop is unrolled
// by four, so the loads of four terms issue ahead of their adds (measured
// faster than a hand-pipelined four-ahead loop with predicated adds: 644
// against 670 cycles per trial on a two-species chain whose exact tier
// decides 1.7% of the trials).
static __device__ __noinline__ int halo_exact_far(const ChainJob* __restrict__ Jg, const double* V,
                                                  const uint32_t* ents, const int16_t* sstart, int lat_off,
                                                  int SZ, int SY, int bcc, int ns, int nsh, int pa, int pb,
                                                  int par_a, int par_b, int sa, int sb, uint32_t wu, int lane) {
  const int nc = 4 * nsh;
  double part[2] = {0.0, 0.0};
#pragma unroll 1
  for (int r = 0; r < 2; ++r) {
    const int c = lane + 32 * r;
    double sum = 0.0;
    if (c < nc) {
      const int ev = c / nsh, sh = c - ev * nsh;
      const bool on2 = ev & 1, after = ev >= 2;
      const int base = lat_off + (on2 ? pb : pa);
      const int par = on2 ? par_b : par_a;
      const int cs = (on2 != after) ? sb : sa;
      // Vr[ns * s] = V(cs, s, sh) for the neighbour species s (1-based)
      const double* Vr = V + (cs - 1) + ns * ns * sh - ns;
      const int k1 = sstart[sh + 1];
      // unrolled by four: the loads of four terms issue ahead of their adds
#pragma unroll 4
      for (int k = sstart[sh]; k < k1; ++k)
        sum = __dadd_rn(sum, Vr[ns * halo_nbr_species(ents[k], base, par, SZ, SY, bcc)]);
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

// Log-domain acceptance thresholds: the uphill decision as two integer
// compares of the fixed-point energy change against bounds taken from the
// acceptance word (no exponential of the change).  The reference accepts an uphill move iff u < exp(-beta dE_ref)
// (src/metropolis.F90:802), i.e. iff t > beta dE_ref log2(e) with
// t = -log2(u) = 32 - log2(w) for u = w 2^-32.  With k = beta 2^-S log2(e)
// and the fixed-point dE within band quanta of dE_ref 2^S, the move is
// certainly accepted when dE < (t - e)/k - band and certainly rejected when
// dE > (t + e)/k + band, where e = 1e-4 bounds the error of t as computed
// here (float conversion of w, lg2.approx, the subtraction: together below
// 2e-5 on [0, 32]) with room to spare.  The float products carry a further
// relative 1e-6 and the thresholds are rounded towards the undecided side.
// Between the two, and for w = 0, the exact tier decides.
struct AcceptThresholds {
  int acc_below;  // dE < acc_below: accepted
  int rej_above;  // dE > rej_above: rejected
};

__device__ __forceinline__ AcceptThresholds accept_thresholds(uint32_t w, float inv_k, float band_f) {
  AcceptThresholds T;
  float lw;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(lw) : "f"(__uint2float_rn(w)));
  const float t = 32.0f - lw;
  const float a = __fmul_rn(__fmul_rn(t - 1e-4f, inv_k), 1.0f - 1e-6f) - band_f - 1.0f;
  const float r = __fmul_rn(__fmul_rn(t + 1e-4f, inv_k), 1.0f + 1e-6f) + band_f + 1.0f;
  // fixed-point changes stay within +-2^30: clamp before converting
  T.acc_below = w == 0u ? INT_MIN : __float2int_rd(fminf(a, 1073741824.0f));
  T.rej_above = w == 0u ? INT_MAX : __float2int_ru(fminf(r, 2147483520.0f));
  return T;
}

// A position's two sites as its lane holds them, one word a site:
//   bits 0-17  padded index of the site
//   bit  18    its parity (bcc z & 1, fcc x & 1)
//   bits 19-22 its species
//   bits 23-28 per axis (x, y, z) 1: it has an image one period up, 2: one
//              period down (the cells an accepted swap writes too)
//   bit  29    (site 1) the pair may be within interaction range
constexpr int kSiteIndex = (1 << 18) - 1;
constexpr int kSiteParity = 18, kSiteSpecies = 19, kSiteImages = 23, kSiteNear = 29;
static_assert(kMaxSpecies < 16, "a species takes four bits");

__device__ __forceinline__ int site_species(int v) { return (v >> kSiteSpecies) & 15; }

__device__ __forceinline__ int image_code(int c, int h, int N) { return c < h ? 1 : (c >= N - h ? 2 : 0); }

// The trial that starts at a position, as far as the stream alone decides it.
struct WinTrial {
  int a, b;          // the two sites (species not filled in)
  int d;             // site 2 - site 1 modulo the periods W: x + W1 (y + W2 z)
  AcceptThresholds th;
};

// The sites' doubled-grid coordinates and compact (Y', X') from the
// position's words.
struct PairCoords {
  int ax, ay, az, Ya, Xa, bx, by, bz, Yb, Xb;
};

__device__ __forceinline__ PairCoords pair_coords(const Geom& g, bool bcc, bool nbr, const uint32_t* w) {
  PairCoords c;
  draw_site_halo(g, bcc, w[0], w[1], w[2], c.ax, c.ay, c.az, c.Ya, c.Xa);
  if (nbr) {
    draw_nbr(g, w[3], c.ax, c.ay, c.az, c.bx, c.by, c.bz);
    c.Yb = c.by >> g.ys;
    c.Xb = c.bx >> 1;
  } else {
    draw_site_halo(g, bcc, w[3], w[4], w[5], c.bx, c.by, c.bz, c.Yb, c.Xb);
  }
  return c;
}

__device__ __forceinline__ int pack_site(const HaloGeom& H, bool bcc, int x, int z, int Yc, int Xc) {
  const int par = bcc ? (z & 1) : (x & 1);
  const int img = image_code(Xc, H.hx, H.NX) | image_code(Yc, H.hy, H.NY) << 2 | image_code(z, H.hz, H.NZ) << 4;
  return halo_index(H, z, Yc, Xc) | par << kSiteParity | img << kSiteImages;
}

__device__ __forceinline__ WinTrial win_decode(const Geom& g, const HaloGeom& H, bool bcc, bool nbr,
                                               const uint32_t* w, float inv_k, float band_f) {
  WinTrial T;
  const PairCoords c = pair_coords(g, bcc, nbr, w);
  const int W1 = 2 * g.n1, W2 = 2 * g.n2, W3 = 2 * g.n3;
  int dx = c.bx - c.ax, dy = c.by - c.ay, dz = c.bz - c.az;
  dx += dx < 0 ? W1 : 0;
  dy += dy < 0 ? W2 : 0;
  dz += dz < 0 ? W3 : 0;
  const bool near = (dx <= H.dmx || dx >= W1 - H.dmx) & (dy <= H.dmy || dy >= W2 - H.dmy) &
                    (dz <= H.dmz || dz >= W3 - H.dmz);
  T.d = dx + W1 * (dy + W2 * dz);
  T.a = pack_site(H, bcc, c.ax, c.az, c.Ya, c.Xa) | (near ? 1 << kSiteNear : 0);
  T.b = pack_site(H, bcc, c.bx, c.bz, c.Yb, c.Xb);
  T.th = accept_thresholds(w[nbr ? 4 : 6], inv_k, band_f);
  return T;
}

// One warp per chain.  What bounds it: a chain's trials are one dependent
// sequence, so a trial's latency -- the shuffles that fetch its sites, two
// shared loads (neighbour species, difference table), a redux.sync, the
// decision -- times the longest chain's trials is the launch's time; neither
// issue slots nor shared-memory bandwidth are near their limits.  So all work
// that the stream alone decides is taken off that sequence (trial_window.cuh):
// the sites, their species, the thresholds and the image cells are decoded for
// 32 positions at once, and a trial of two like species is a bit of a mask.
template <int NJ, bool FULL>
__global__ void __launch_bounds__(32) metropolis_halo_kernel(const ChainJob* __restrict__ jobs) {
  extern __shared__ __align__(16) unsigned char smem[];
  extern __shared__ int32_t s_i32[];
  extern __shared__ int8_t s_i8[];
  const ChainJob* Jg = jobs + blockIdx.x;
  if (Jg->status && *Jg->status != 0) return;  // the chain's input was flagged: no trial runs
  const Geom g = Jg->g;
  const HaloGeom H = Jg->hg;
  const int lane = threadIdx.x;
  __shared__ unsigned long long s_t_start;  // kept out of registers
  if (lane == 0) s_t_start = global_ns();
  const WindowLayout L = window_layout(g, H);
  uint32_t* mt = reinterpret_cast<uint32_t*>(smem + L.mt);
  uint32_t* old = mt + kMTN;
  uint32_t* tw = old + kOldWords;
  double* V = reinterpret_cast<double*>(smem + L.V);
  uint32_t* ents = reinterpret_cast<uint32_t*>(smem + L.ents);
  int16_t* sstart = reinterpret_cast<int16_t*>(smem + L.sstart);
  int32_t* I = reinterpret_cast<int32_t*>(smem + L.I);
  int8_t* lat = reinterpret_cast<int8_t*>(smem + L.lat);

  // ---- stage state ------------------------------------------------------
  const int nsp = g.ns + 1;
  const int nI = nsp * nsp * g.nsh * (1 + nsp), nV = g.ns * g.ns * g.nsh;
  const uint32_t* rng = Jg->rng;
  for (int i = lane; i < kMTN; i += 32) mt[i] = rng[i];
  for (int i = lane; i < nI; i += 32) I[i] = Jg->F[i];
  for (int i = lane; i < nV; i += 32) V[i] = Jg->V[i];
  for (int i = lane; i < g.z; i += 32) ents[i] = Jg->entries[i];
  for (int i = lane; i <= g.nsh; i += 32) sstart[i] = Jg->shell_start[i];
  __syncwarp();
  halo_fill(g, H, Jg->lat, lat, lane);
  HaloPlan<NJ> P;
  make_halo_plan<NJ>(g, H, ents, lane, P);
  const int lat_off = (int)L.lat;
  const int I_off = (int)(L.I / 4);
  const int D_abs = I_off + L.D_off;
  const bool bcc = g.lattice == kBcc;
  const bool nbr_swap = Jg->nbr_swap != 0;
  const bool on_b = lane >= 16;  // lanes 0-15 sum site 1's neighbours, 16-31 site 2's
  // this lane's entries modulo the periods, as the displacement site 2 -
  // site 1 that makes the entry's neighbour the other site
  int32_t* ecan = s_i32 + L.ecan / 4;
  {
    const int W1 = 2 * g.n1, W2 = 2 * g.n2, W3 = 2 * g.n3;
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int k = (lane & 15) + 16 * j;
      int e = -1;  // no entry: matches no displacement
      if (k < g.z) {
        int dx, dy, dz, sh;
        unpack_entry(ents[k], dx, dy, dz, sh);
        dx = on_b ? -dx : dx;
        dy = on_b ? -dy : dy;
        dz = on_b ? -dz : dz;
        e = (dx < 0 ? dx + W1 : dx) + W1 * ((dy < 0 ? dy + W2 : dy) + W2 * (dz < 0 ? dz + W3 : dz));
      }
      ecan[32 * j + lane] = e;
    }
  }
  const int band = Jg->band;
  const float inv_k = 1.0f / Jg->beta_q_l2, band_f = (float)band;
  const int n_base = nbr_swap ? 4 : 6;
  const int nt = (int)Jg->n_trials;
  // lanes 0-7 write site 1's cells of an accepted swap, lanes 8-15 site 2's:
  // lane c of eight takes the image axes that its bits name
  const int img_axes = ((lane & 1) ? 3 : 0) | ((lane & 2) ? 12 : 0) | ((lane & 4) ? 48 : 0);
  // 32-bit tallies (a launch runs fewer than 2^31 trials per chain, see
  // launch_metropolis_halo); the words drawn follow from them: n_base per
  // trial plus the uniforms
  unsigned int b_eval = 0, b_acc = 0, b_exact = 0;
  unsigned int c_fp64 = 0, c_cr = 0;

  // ---- the stream -----------------------------------------------------------
  const int pos0 = (int)rng[kMTN];
  MtRoll R = {pos0, 0, false};
#pragma unroll 1
  for (int i = 0; i < kLookAhead / kWin; ++i) mt_roll(mt, old, tw, R, lane);
  WinTrial cur, nxt;
  unsigned int n_win = 0;  // windows begun
  int tb = -kWin;          // the window's place in the tempered ring
  unsigned diff = 0;       // positions whose two species differ
  auto decode_next = [&](int at) {
    uint32_t w[7];
#pragma unroll
    for (int i = 0; i < 7; ++i) w[i] = tw[at + lane + i];
    nxt = win_decode(g, H, bcc, nbr_swap, w, inv_k, band_f);
  };
  decode_next(0);
  // the next window becomes the current one: its species are read, the one
  // after it is decoded and 32 more words are generated
  auto advance = [&]() {
    cur = nxt;
    tb = (tb + kWin) & (kTwRing - 1);
    const int sa = s_i8[lat_off + (cur.a & kSiteIndex)], sb = s_i8[lat_off + (cur.b & kSiteIndex)];
    decode_next((tb + kWin) & (kTwRing - 1));
    mt_roll(mt, old, tw, R, lane);
    cur.a |= sa << kSiteSpecies;
    cur.b |= sb << kSiteSpecies;
    diff = __ballot_sync(kFull, sa != sb);
    ++n_win;
  };
  int o = 0;  // the next trial's position in the window
  advance();

  for (int t = 0; t < nt; ++t) {
    if (o >= kWin) {
      o -= kWin;
      advance();
    }
    if (!((diff >> o) & 1u)) {
      // same species: accepted without an energy evaluation or a draw
      ++b_acc;
      o += n_base;
      continue;
    }
    ++b_eval;
    const int a = __shfl_sync(kFull, cur.a, o), b = __shfl_sync(kFull, cur.b, o);
    const int acc_below = __shfl_sync(kFull, cur.th.acc_below, o);
    const int rej_above = __shfl_sync(kFull, cur.th.rej_above, o);
    const int mine = on_b ? b : a;
    const int base = lat_off + (mine & kSiteIndex);
    const bool par = (mine >> kSiteParity) & 1;
    const int so = site_species(mine), sn = site_species(on_b ? a : b);
    const int K = g.nsh * nsp;
    const int rowD = D_abs + (so * nsp + sn) * K;
    int acc = 0;
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int s = s_i8[base + (par ? P.d1[j] : P.d0[j])];
      const int v = s_i32[rowD + P.shp[j] + s];
      acc += (FULL || ((P.valid >> j) & 1u)) ? v : 0;
    }
    const bool near = (a >> kSiteNear) & 1;
    if (near) {
      // an entry whose neighbour is the other site: that site holds our old
      // species after the swap, not its own
      const int d = __shfl_sync(kFull, cur.d, o);
      const int rowN = I_off + sn * K;
#pragma unroll
      for (int j = 0; j < NJ; ++j)
        if (ecan[32 * j + lane] == d) acc += s_i32[rowN + P.shp[j] + so] - s_i32[rowN + P.shp[j] + sn];
    }
    const int dE = __reduce_add_sync(kFull, acc);
    int consumed = n_base;
    int accept = -1;
    if (dE < -band) {
      accept = 1;
    } else if (dE > band) {
      consumed = n_base + 1;
      accept = dE < acc_below ? 1 : (dE > rej_above ? 0 : -1);
    }
    if (accept < 0) {
      ++b_exact;
      const uint32_t* w = tw + tb + o;
      const uint32_t wu = w[n_base];
      const int sa = site_species(a), sb = site_species(b);
      int r;
      if (near) {
        const PairCoords c = pair_coords(g, bcc, nbr_swap, w);
        const HaloLat hl = {g.sz, g.sy, H.origin, H.SZ, H.SY, lat_off};
        r = halo_exact_decision(Jg, hl, V, ents, sstart, c.ax, c.ay, c.az, c.az * g.sz + c.Ya * g.sy + c.Xa,
                                c.bx, c.by, c.bz, c.bz * g.sz + c.Yb * g.sy + c.Xb, sa, sb, lane, wu);
      } else {
        r = halo_exact_far(Jg, V, ents, sstart, lat_off, H.SZ, H.SY, bcc, g.ns, g.nsh, a & kSiteIndex,
                           b & kSiteIndex, (a >> kSiteParity) & 1, (b >> kSiteParity) & 1, sa, sb, wu, lane);
      }
      accept = r & 1;
      consumed = (r & 2) ? n_base + 1 : n_base;
      c_fp64 += (r >> 2) & 1;
      c_cr += (r >> 3) & 1;
    }
    if (accept) {
      ++b_acc;
      const int sa = site_species(a), sb = site_species(b);
      const int ia = a & kSiteIndex, ib = b & kSiteIndex;
      // the cells of the swapped sites: lane c of eight shifts along its axes
      const int v = lane < 8 ? a : b;
      const int code = (v >> kSiteImages) & img_axes;
      int cell = v & kSiteIndex;
      cell += (code & 1) ? H.NX : ((code & 2) ? -H.NX : 0);
      cell += (code & 4) ? H.NY * H.SY : ((code & 8) ? -H.NY * H.SY : 0);
      cell += (code & 16) ? H.NZ * H.SZ : ((code & 32) ? -H.NZ * H.SZ : 0);
      // every axis of this lane has an image
      const int has = code | (code >> 1);
      if (lane < 16 && (has & 0x15) == (img_axes & 0x15)) s_i8[lat_off + cell] = (int8_t)(lane < 8 ? sb : sa);
      // the window's positions that name either site
      const int xa = cur.a & kSiteIndex, xb = cur.b & kSiteIndex;
      const int flip = (sa ^ sb) << kSiteSpecies;
      if (xa == ia || xa == ib) cur.a ^= flip;
      if (xb == ia || xb == ib) cur.b ^= flip;
      diff = __ballot_sync(kFull, ((cur.a ^ cur.b) >> kSiteSpecies) & 15);
      __syncwarp();  // the written cells are read by the next trial's lanes
    }
    o += consumed;
  }

  // ---- write back ---------------------------------------------------------
  __syncwarp();
  const unsigned long long words = (unsigned long long)kWin * (n_win - 1) + (unsigned long long)o;
  halo_store(g, H, lat, Jg->lat, lane);
  mt_roll_store(mt, old, tw, R, pos0, words, (unsigned long long)kWin * n_win + kLookAhead, Jg->rng, lane);
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

template <int NJ, bool FULL>
static void launch_halo_nj(const ChainJob* d_jobs, int n_jobs, uint32_t smem_bytes,
                           cudaStream_t stream) {
  cudaFuncSetAttribute(metropolis_halo_kernel<NJ, FULL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)smem_bytes);
  BRAWL_CARVEOUT((metropolis_halo_kernel<NJ, FULL>));
  metropolis_halo_kernel<NJ, FULL><<<n_jobs, 32, smem_bytes, stream>>>(d_jobs);
}

void launch_metropolis_halo(const ChainJob* d_jobs, int n_jobs, uint32_t smem_bytes, int min_z,
                            int max_z, cudaStream_t stream) {
  if (n_jobs <= 0) return;
  const int nj = lane_entries_for(max_z);
  // every chain with z = 64 (bcc, 6 shells): no lane entry to mask
  const bool full = min_z == max_z && max_z == 16 * nj;
  switch (nj) {
    case 2: launch_halo_nj<2, false>(d_jobs, n_jobs, smem_bytes, stream); break;
    case 4:
      if (full) launch_halo_nj<4, true>(d_jobs, n_jobs, smem_bytes, stream);
      else launch_halo_nj<4, false>(d_jobs, n_jobs, smem_bytes, stream);
      break;
    case 6: launch_halo_nj<6, false>(d_jobs, n_jobs, smem_bytes, stream); break;
    case 8: launch_halo_nj<8, false>(d_jobs, n_jobs, smem_bytes, stream); break;
    default: launch_halo_nj<11, false>(d_jobs, n_jobs, smem_bytes, stream); break;
  }
}

void preload_halo_kernels() {
  cudaFuncAttributes a;
  cudaFuncGetAttributes(&a, metropolis_halo_kernel<2, false>);
  cudaFuncGetAttributes(&a, metropolis_halo_kernel<4, false>);
  cudaFuncGetAttributes(&a, metropolis_halo_kernel<4, true>);
  cudaFuncGetAttributes(&a, metropolis_halo_kernel<6, false>);
  cudaFuncGetAttributes(&a, metropolis_halo_kernel<8, false>);
  cudaFuncGetAttributes(&a, metropolis_halo_kernel<11, false>);
}

}  // namespace brawl
