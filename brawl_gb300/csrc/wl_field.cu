// wl_field.cu -- Wang-Landau sweeps of walkers whose sites' fields fit in
// shared memory (field_engine.cuh): sweeps() of src/wang-landau.F90:539-632 as
// wang_landau.cu's wl_sweep_kernel runs it, trial for trial, on the same state.
//
// A trial's bin follows from the walker's energy and the trial's change; its
// test compares log(u) with ln g of the two bins, and every trial adds f to ln g
// of the bin it ends in.  While the walker stays where it is, all that changes
// is ln g of its own bin, by f a trial, so the trials of two windows are decided
// at once: like pairs and certain rejections are passed, and so are trials
// whose bin is outside the window (those draw no uniform).  The first other
// trial is taken on its own: accepted moves are logged and their FP64 energies
// summed later (lazy_exact.cuh), and a test or a bin that the intervals do not
// settle takes the exact values, as in wl_sweep_kernel.
#include <climits>

#include "field_engine.cuh"
#include "lazy_exact.cuh"
#include "wl_kernels.cuh"

namespace brawl {

// Shared memory after the fields': the window's ln g and histogram, ln g in
// fixed point, its open store flags, and the log.
struct WlFieldLayout {
  uint32_t lng, hist, lq, sopen, lazy, total;
};

__host__ __device__ inline WlFieldLayout wl_field_layout(const Geom& g, const FieldGeom& f, int nb, int cap) {
  WlFieldLayout L;
  L.lng = align_up(field_layout(g, f).total, 16);
  L.hist = L.lng + (uint32_t)nb * 8;
  L.lq = L.hist + (uint32_t)nb * 8;
  L.sopen = L.lq + (uint32_t)nb * 8;
  L.lazy = align_up(L.sopen + (uint32_t)nb, 16);
  L.total = L.lazy + (cap > 0 ? lazy_bytes(g, cap) : 0);
  return L;
}

uint32_t wl_field_smem_bytes(const Geom& g, const FieldGeom& f, int nb, int cap) {
  return wl_field_layout(g, f, nb, cap).total;
}

namespace {

constexpr int kUnsettled = INT_MIN;

// What the team shares of two windows (twice: one pair is written while the
// other is read): per position the walk from it (bits 0-7 where it ends, 32 and
// more past the window; 8-15 trials passed; 16-23 like pairs among them; 24-31
// trials outside the window), the trial's change and species (as stored, site
// 2's from bit 8; bit 16: certainly accepted), and its bin.
struct WlShare {
  unsigned walk[2][2 * kWin];
  int2 pos[2][2 * kWin];
  int bin[2][2 * kWin];
  double e_sw;
  int verdict;
};
static_assert(own_bytes<FieldEnd, WlShare>() == kWlFieldOwn, "what the layout leaves room for");

// field_walk (field_engine.cuh) for the masks of trials that draw n_base + 1
// words and n_base words.
__device__ __forceinline__ unsigned wl_walk(unsigned like, unsigned long_m, unsigned short_m, int lane, int n_base,
                                            bool nbr) {
  unsigned path = 1u << lane;
#pragma unroll
  for (int i = 0; i < 5; ++i) path |= ((path & short_m) << n_base) | ((path & long_m) << (n_base + 1));
  if (nbr) {
    path |= ((path & short_m) << n_base) | ((path & long_m) << (n_base + 1));
    path |= ((path & short_m) << n_base) | ((path & long_m) << (n_base + 1));
  }
  const unsigned n_long = __popc(path & long_m), n_short = __popc(path & short_m), n_like = __popc(path & like);
  return ((unsigned)lane + (n_long + n_short) * (unsigned)n_base + n_long) | (n_long + n_short) << 8 | n_like << 16 |
         n_short << 24;
}

// bin_index (src/wang-landau.F90:515-523), as in wang_landau.cu.
__device__ __forceinline__ int field_bin_index(double E, double e1, double range, int bins) {
  const double t = __dmul_rn(__ddiv_rn(__dsub_rn(E, e1), range), (double)bins);
  if (!(t > -1.0e9 && t < 1.0e9)) return t < 0.0 ? -1000000000 : 1000000000;
  return (int)t + 1;
}

// ln g in fixed point, 2^-32, for the tests that its nearness does not matter
// to: the sums and differences cost a warp no FP64.  A trial adds f's rounding
// to it (2^-33 at most) and what the double's own sum rounds.  A value past 2^18
// (or not a number) has none, and its tests take the exact values.
constexpr long long kNoFixed = LLONG_MIN;
constexpr double kFixedMost = 262144.0;  // 2^18: differences in 2^-12 fit 32 bits

__device__ __forceinline__ long long lng_fixed(double v) {
  return fabs(v) < kFixedMost ? __double2ll_rn(__dmul_rn(v, 4294967296.0)) : kNoFixed;
}

// The doubles 0 to 16 (a conversion takes the FP64 pipe as long as a sum).
static __constant__ double cCount[17] = {0.0, 1.0, 2.0,  3.0,  4.0,  5.0,  6.0,  7.0, 8.0,
                                         9.0, 10.0, 11.0, 12.0, 13.0, 14.0, 15.0, 16.0};

// k times v = v + f, each rounded, as the reference adds them.  Within one
// binade v is a multiple of its ulp and every sum rounds f to the same multiple
// f_r of it, unless f lies halfway between two (then the neighbours' parity
// decides): v + k f_r is that sequence's end, exactly.
__device__ __forceinline__ double add_times(double v, double f, int k) {
  if (k >= 4 && k <= 16) {
    const double fr = __dsub_rn(__dadd_rn(v, f), v);
    const double end = __fma_rn(cCount[k], fr, v), off = __dsub_rn(f, fr);
    const int ev = __double2hiint(v) & 0xfff00000, ee = __double2hiint(end) & 0xfff00000;
    // half an ulp of v (v a normal number well above the smallest), compared by
    // the bits
    const long long half = (long long)((ev & 0x7ff00000) - (53 << 20)) << 32;
    if (__double2hiint(f) >= 0 && ev >= 0 && ev == ee && (ev & 0x7ff00000) > (60 << 20) && (ev & 0x7ff00000) < 0x7ff00000 &&
        (__double_as_longlong(off) & 0x7fffffffffffffffll) < half)
      return end;
  }
  for (int i = 0; i < k; ++i) v = __dadd_rn(v, f);
  return v;
}

}  // namespace

// One walker per block, the roles of metropolis_field_kernel; the team's third
// warp also keeps the books: ln g and the histogram are added to one trial at a
// time, in order (each add rounds), beside the other warps' next decisions.
//
// A walker's trials depend on one another, so its own chain of decisions bounds
// it: a pair of windows takes some 700 cycles to decide and walk and an accepted
// move 800 more (its log entry, the fields' update), against some
// 2,900 a trial in wl_sweep_kernel, which gathers both sites' neighbours for
// each.  FP64 is kept out of the decisions (a dependent FP64 add takes a warp 64
// cycles): bins from a float interval, tests from ln g's fixed-point copy.
// Measured on 128 walkers of bcc 12^3, four species, four shells, 10^4 trials: a
// call takes 11 to 12 ms with wl_sweep_kernel and 2.7 to 4.7 ms here (walkers
// that accept 38% to 55% of their trials).  16 warps a block would leave each too
// few registers (spills), hence 8.
template <int NJ, int R>
__global__ void __launch_bounds__(256, 1) wl_field_kernel(WlWalker* __restrict__ walkers) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ FieldEnd end;
  __shared__ __align__(16) WlShare S;
  WlWalker& W = walkers[blockIdx.x];
  const ChainJob& J = W.job;
  const Geom g = J.g;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned long long t_start = global_ns();
  const FieldLayout L = field_layout(g, J.fg);
  const int start = W.start, nb = W.end - start + 1;
  const WlFieldLayout WL = wl_field_layout(g, J.fg, nb, W.field_cap);
  double* lng = reinterpret_cast<double*>(smem + WL.lng);
  double* hist = reinterpret_cast<double*>(smem + WL.hist);
  long long* lq = reinterpret_cast<long long*>(smem + WL.lq);
  uint8_t* sopen = smem + WL.sopen;
  for (int i = tid; i < nb; i += blockDim.x) {
    const double v = W.lng[start - 1 + i];
    lng[i] = v;
    lq[i] = lng_fixed(v);
    hist[i] = W.hist[i];
    sopen[i] = W.store ? W.store_open[start - 1 + i] : (uint8_t)0;
  }
  if (tid == 0) end.done = 0;
  field_stage(J, g, L, smem, tid, blockDim.x);
  if (warp < 8 && (warp & 2) == 0) {
    // A's last word: log(u) as a float (within 1e-5 of it); B's third: the word
    field_produce(J, g, L, smem, &end, (warp & 1) + (warp >> 1), lane, [](uint32_t w) {
      float lw;
      asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(lw) : "f"(__uint2float_rn(w)));
      return make_int2(__float_as_int((lw - 32.0f) * 0.693147182f), (int)w);
    });
  } else if (warp < 8) {
    const int who = (warp & 1) + (warp >> 2) * 2, tt = who * 32 + lane;
    const bool second = tt >= kFieldHalf;
    // the entries are symmetric: the sites that have a swapped site as a
    // neighbour are its own neighbours
    FieldPlan<NJ> P;
    field_plan<NJ>(g, L, smem, tt, P, 1);
    const LazyLog LG = lazy_layout(g, smem + WL.lazy, W.field_cap);
    const double* V = reinterpret_cast<const double*>(smem + FieldLayout::kV);
    const int16_t* sstart = reinterpret_cast<const int16_t*>(smem + L.sstart);
    const int distinct = J.fg.distinct;
    const bool nbr = J.nbr_swap != 0;
    const int n_base = nbr ? 4 : 6;
    const int nt = (int)W.n_trials;
    const int band = J.band, ns = g.ns, r = field_stride(ns), stride = 4 * r, per = g.nsh * stride, z = g.z;
    const int g_at = (int)L.g - 4;  // species 1 (0 as stored) has no field: its loads are read past
    const double e1 = W.e1, range = W.range, f = W.wl_f;
    // (the float's roundings, and the quotients', within 1e-5 of them)
    const float ff = __double2float_rn(f), f_lo = ff / (float)(n_base + 1) * (1.0f - 1.0e-5f),
                f_hi = ff / (float)n_base * (1.0f + 1.0e-5f);
    const int bins = W.bins, last = W.end;
    const double rbins = __ddiv_rn((double)bins, range);
    const int period = W.hist_period;
    const double q1 = ldexp(1.0, -W.S);  // one fixed-point quantum
    const float qrf = __double2float_rn(__dmul_rn(q1, rbins));
    // e_ex: the reference's e_unswapped before the n_log logged moves; after
    // them it lies in e_ex + [Dlo, Dhi] quanta
    double e_ex = (W.i0 > 0 && W.e_state) ? *W.e_state : (W.e0_src ? *W.e0_src : W.e0);
    long long Dlo = 0, Dhi = 0;
    // the coordinate of e_ex on the bins, whole and fraction, and one more move's
    // interval without its change (base), with bin_of's constants
    int t0 = 0;
    float t0_frac = 0.0f, wide = 0.0f;
    long long base_lo = 0, base_hi = 0;
    int lo32 = 0;
    // `small`: the interval fits 32 bits with any change.  A logged update, and the
    // next one, round by 2^-53 of twice the energy at most, under a quantum while
    // the energy stays under 2^51 quanta; where it does not, or the coordinate is
    // far out, nothing is settled (`lost`).
    bool small = false, lost = false;
    auto bounds = [&]() {
      base_lo = Dlo - band - 1;
      base_hi = Dhi + band + 1;
      small = base_lo > -(1ll << 30) && base_hi < (1ll << 30);
      lo32 = (int)base_lo;
      wide = __fmul_ru(__int2float_ru((int)(base_hi - base_lo)), qrf);
    };
    auto rebase = [&]() {
      const double t = __dmul_rn(__dsub_rn(e_ex, e1), rbins);
      lost = quanta_bound(e_ex, W.S) >= (1ll << 51) || !(fabs(t) < 5.0e8);
      const double whole = lost ? 0.0 : floor(t);
      t0 = (int)whole;
      t0_frac = __double2float_rn(__dsub_rn(t, whole));
      Dlo = Dhi = 0;
      bounds();
    };
    rebase();
    // The bin (int(t) + 1, as bin_index) after change dE, when the interval lies
    // in one bin.  The ends' offsets from t0 are t0_frac + p and that + wide.  Their
    // errors: 6e-8 of t0_frac and 1e-7 of t's own (5e-16 of at most 5e8, twice),
    // 1.8e-7 |p| and |wide| (the floats' products), 6e-8 of the sums; m is at
    // least that.  int() truncates: below zero, where t < 0, it is one up.
    auto bin_of = [&](int dE, int& b) {
      const float p = __fmul_rn(__int2float_rn(lo32 + dE), qrf);
      const float t = __fadd_rn(t0_frac, p);
      const float m = __fmaf_rn(3.0e-7f, fabsf(p) + wide, 8.0e-7f);
      const float lo = floorf(__fsub_rd(t, m)), hi = floorf(__fadd_ru(t, wide + 2.0f * m));
      const int w = t0 + (int)lo;
      b = w < 0 ? w + 2 : w + 1;
      return lo == hi && small && fabsf(lo) < 1.0e9f && !lost;
    };
    int n_log = 0;
    int ibin = field_bin_index(e_ex, e1, range, bins);
    int status = (ibin < start || ibin > last) ? kStatusWalkerOutsideWindow : kStatusOk;
    unsigned c_eval = 0, c_exp = 0, c_exact = 0, n_acc = 0;
    DecideStats st = {0u, 0u};
    const bool stored = W.store != nullptr;
    int until = period > 0 ? period - (int)(W.i0 % period) : 0;
    auto flush = [&]() {
      if (n_log == 0) return;
      lazy_sites_any<4>(g, V, sstart, LG, n_log, kFoldWangLandau, tt, kFieldTeam);
      team_sync();
      const double before = e_ex;
      e_ex = lazy_fold(LG, n_log, e_ex, kFoldWangLandau);
      if (!in_quanta(e_ex, before, Dlo, Dhi, q1)) status = kStatusBandViolated;
      n_log = 0;
      rebase();
    };
    // histogram ticks among the next k trials
    auto ticks = [&](int k) {
      int h = 0;
      if (period <= 0) return 0;
      for (; k >= until; until = period) {
        k -= until;
        ++h;
      }
      until -= k;
      return h;
    };
    // config_per_bin(b) = config the first time the bin is sampled
    // (src/wang-landau.F90:605-610)
    auto store = [&](int b) {
      if (!sopen[b - start]) return;
      int8_t* dst = W.store + (size_t)(b - 1) * (size_t)g.n_sites;
      for (int i = tt; i < g.n_sites; i += kFieldTeam) dst[i] = (int8_t)((smem[L.lat + i] >> 2) + 1);
      team_sync();
      if (tt == 0) sopen[b - start] = 0;
      team_sync();
    };
    // the books: k trials and h histogram ticks in bin b (the third warp's)
    auto book = [&](int b, int k, int h) {
      if (lane == 0) {
        lng[b - start] = add_times(lng[b - start], f, k);
        for (int i = 0; i < h; ++i) hist[b - start] = __dadd_rn(hist[b - start], 1.0);
      }
      __syncwarp();
    };
    unsigned n_win = 0;  // windows passed
    int o = 0, t = 0;    // the next trial's position in the window; trials done
    int slot = 0;        // the window's place in the record ring
    unsigned have = 0;   // the last part waited for
    int flip = 0;        // the shared pair in use
    auto after = [&](int at, int by) { return at + by >= kFieldRing ? at + by - kFieldRing : at + by; };
    // k = 0, 1 or 2 windows on; the window after the next one is at hand
    auto pass_windows = [&](int k) {
      const unsigned before = n_win / kFieldMakers;
      n_win += k;
      slot = after(slot, k * kWin);
      if (n_win / kFieldMakers != before) used_arrive((int)(before & 1u));
      if ((n_win + 1) / kFieldMakers != have) {
        ++have;
        made_wait((int)(have & 1u));
      }
    };
    made_wait(0);
    // ln g of the walker's bin in fixed point (lq holds the other bins'), and f
    const long long fq = fabs(f) < 65536.0 ? __double2ll_rn(__dmul_rn(f, 4294967296.0)) : 0;
    const bool f_ok = f >= 0.0 && f < 65536.0;
    long long li = status == kStatusOk && f_ok ? lq[ibin - start] : kNoFixed;
    // k trials' f added; past kFixedMost there is no fixed point any more
    auto plus = [&](long long l, int k) {
      const long long v = l + fq * k;
      return !f_ok || l == kNoFixed || v >= (1ll << 50) ? kNoFixed : v;
    };
    while (t < nt && status == kStatusOk) {
      if (who < 2) {
        const int4 a = *reinterpret_cast<const int4*>(smem + FieldLayout::kA + (after(slot, kWin * who) + lane) * 16);
        const int sa = smem[L.lat + a.x], sb = smem[L.lat + a.y];
        const unsigned char* ga = smem + g_at + a.x * stride;
        const unsigned char* gb = smem + g_at + a.y * stride;
        const int ab = *reinterpret_cast<const int32_t*>(ga + sb), bb = *reinterpret_cast<const int32_t*>(gb + sb);
        const int ba = *reinterpret_cast<const int32_t*>(gb + sa), aa = *reinterpret_cast<const int32_t*>(ga + sa);
        const int met = *reinterpret_cast<const int32_t*>(smem + a.z + sa * ns + sb);
        const int dE = (sb ? ab - bb : 0) + (sa ? ba - aa : 0) + met;
        // the bin; a like pair's is the walker's
        const bool same = sa == sb;
        int jbin;
        const bool settled = bin_of(dE, jbin);
        jbin = same ? ibin : jbin;
        const unsigned jn = (unsigned)(jbin - start);
        const bool inside = jn < (unsigned)nb;
        // the test log(u) < li - lj, li growing by f with each trial passed
        // before this one: between dist/(n_base + 1) and dist/n_base of them.
        // m covers the difference's 2^-12, the floats of log(u) and of the sums,
        // and what lng_fixed's sums may be off by after t trials (2^-33 and 2^-36
        // each)
        const long long lj = lq[inside ? jn : 0u];
        const bool known = li != kNoFixed && lj != kNoFixed;
        const float d = (float)(int)((li - lj) >> 20) * (1.0f / 4096.0f);
        const float lu = __int_as_float(a.w);
        const float dist = fmaxf((float)(lane + kWin * who - o), 0.0f);
        const float m = 6.0e-4f + __fmaf_rn(1.0e-6f, fabsf(d), 1.5e-10f * (float)t);
        const bool own = jbin == ibin;  // li - li: accepted
        const bool mine = settled && inside && !same;
        const bool sure = mine && (own ? li != kNoFixed : (known && lu > -100.0f && lu < __fmaf_rn(f_lo, dist, d) - m));
        const bool rej = mine && !own && known && lu > __fmaf_rn(f_hi, dist, d) + m;
        const bool out = settled && !inside;
        const bool finite = li != kNoFixed;
        const unsigned like_m = __ballot_sync(kFull, same && finite);
        const unsigned long_m = like_m | __ballot_sync(kFull, rej);
        const unsigned short_m = __ballot_sync(kFull, out);
        S.pos[flip][tt] = make_int2(dE, sa | sb << 8 | (sure ? 1 << 16 : 0));
        S.bin[flip][tt] = settled || same ? jbin : kUnsettled;
        S.walk[flip][tt] = wl_walk(like_m, long_m, short_m, lane, n_base, nbr);
      }
      team_sync();
      const unsigned w0 = S.walk[flip][o];
      const int o0 = (int)(w0 & 0xffu);
      const unsigned w1 = o0 >= kWin ? S.walk[flip][o0] : 0u;
      const unsigned w = w0 + w1;  // (the counts; the positions apart)
      int k = (int)((w >> 8) & 0xffu), n_like = (int)((w >> 16) & 0xffu), n_out = (int)(w >> 24);
      const int e = o0 >= kWin;
      const int p = e ? (int)(w1 & 0xffu) : o0;
      int windows = e + (p >= kWin), next_o = p & (kWin - 1);
      bool event = p < kWin;
      if (k >= nt - t) {
        // the run ends among the passed trials: stepped through one by one
        event = false;
        k = n_like = n_out = windows = 0;
        next_o = o;
        for (; k < nt - t; ++k) {
          const int at = next_o + kWin * windows;
          const int2 v = S.pos[flip][at];
          const int b = S.bin[flip][at];
          const bool like = (v.y & 0xff) == ((v.y >> 8) & 0xff), in = b >= start && b <= last;
          n_like += like;
          n_out += !in;
          next_o += n_base + (int)in;
          if (next_o >= kWin) {
            next_o -= kWin;
            ++windows;
          }
        }
      }
      t += k;
      li = plus(li, k);
      if (who == 3) {  // the tallies
        c_eval += k - n_like;
        c_exp += k - n_out;
        n_acc += n_like;
      }
      int h = 0;
      if (who == 2 || stored) h = ticks(k);
      if (stored && h > 0) store(ibin);
      if (!event) {
        if (who == 2) book(ibin, k, h);
        flip ^= 1;
        o = next_o;
        pass_windows(windows);
        continue;
      }
      // ---- a trial of its own -----------------------------------------------
      const int at = after(slot, kWin * e) + p;
      const int4 a = *reinterpret_cast<const int4*>(smem + FieldLayout::kA + at * 16);
      const int4 q = *reinterpret_cast<const int4*>(smem + FieldLayout::kB + at * 16);
      const int2 v = S.pos[flip][kWin * e + p];
      int jbin = S.bin[flip][kWin * e + p];
      const int s1 = v.y & 0xff, s2 = (v.y >> 8) & 0xff;
      const bool differ = s1 != s2;
      const long long dE = v.x;
      bool exact_done = false;
      double e_sw = 0.0;
      ++t;
      c_eval += differ;
      if (jbin == kUnsettled && n_log > 0) {
        // the logged moves' exact energy may settle it
        flush();
        int b = 0;
        if (bin_of(v.x, b)) jbin = b;
      }
      if (jbin == kUnsettled) {
        ++c_exact;
        exact_done = true;
        if (who == 0) {
          const double2 pr = field_exact_pair(field_exact_setup(g, L), q.x, q.y, a.x, a.y, (s1 >> 2) + 1,
                                              (s2 >> 2) + 1, lane);
          // e_swapped = e_unswapped - pair_unswapped + pair_swapped
          if (lane == 0) S.e_sw = __dadd_rn(__dsub_rn(e_ex, pr.x), pr.y);
        }
        team_sync();
        e_sw = S.e_sw;
        jbin = field_bin_index(e_sw, e1, range, bins);
      }
      const bool inside = jbin >= start && jbin <= last;
      int accept = (v.y >> 16) & 1;
      if (inside) ++c_exp;
      if (inside && !accept) {
        if (who == 2) {
          book(ibin, k, h);
          k = h = 0;
          const int verdict = log_u_lt((uint32_t)q.z, __dsub_rn(lng[ibin - start], lng[jbin - start]), st);
          if (lane == 0) S.verdict = verdict;
        }
        team_sync();
        accept = *(volatile int*)&S.verdict;
      }
      n_acc += accept;
      next_o = p + n_base + (int)inside;
      const int from = ibin;
      const long long l_from = li;
      li = plus(accept && jbin != ibin ? lq[jbin - start] : li, 1);
      if (accept) ibin = jbin;
      if (accept && differ) {
        int at_n[NJ];
        field_sites<NJ>(smem, P, second ? q.y : q.x, at_n);
        if (exact_done) {
          e_ex = e_sw;  // the log is empty here
          rebase();
        } else {
          // logged: the species of both sites' neighbours as they are, the
          // other site marked
          uint8_t* rec = LG.codes + (size_t)n_log * 2 * z + (second ? z : 0) + (tt & (kFieldHalf - 1));
          const int other = second ? a.x : a.y, s_other = second ? s1 : s2;
#pragma unroll
          for (int j = 0; j < NJ; ++j)
            if ((P.valid >> j) & 1) {
              const bool met = at_n[j] == other;
              const int s = met ? s_other >> 2 : smem[L.lat + at_n[j]] >> 2;
              rec[kFieldHalf * j] = (uint8_t)(s + 1 + (met ? kLazyPartner : 0));
            }
          if (tt == 0) {
            LG.spec[2 * n_log] = (int8_t)((s1 >> 2) + 1);
            LG.spec[2 * n_log + 1] = (int8_t)((s2 >> 2) + 1);
          }
          // (its change to band quanta, and its update's rounding)
          Dlo += dE - band - 1;
          Dhi += dE + band + 1;
          ++n_log;
          bounds();
        }
        if (tt == 0) {
          smem[L.lat + a.x] = (unsigned char)s2;
          smem[L.lat + a.y] = (unsigned char)s1;
        }
        const int row = (int)L.U + ((second ? s2 * ns + s1 : s1 * ns + s2) >> 2) * per;
        field_update<NJ, R>(L, smem, P, distinct, r, at_n, row, q.w != 0, second);
      }
      if (tt == kFieldHalf && ibin != from) lq[from - start] = l_from;
      team_sync();
      int h1 = 0;
      if (who == 2 || stored) h1 = ticks(1);
      if (stored && h1 > 0) store(ibin);
      // the books of the bin it was in and of the one it is in, beside the next
      // decisions
      if (who == 2) {
        if (ibin != from) {
          book(from, k, h);
          book(ibin, 1, h1);
        } else {
          book(ibin, k + 1, h + h1);
        }
      }
      if (n_log == LG.cap) flush();
      pass_windows(e + (next_o >= kWin));
      o = next_o & (kWin - 1);
    }
    flush();
    // the makers have made, or are making, the part after this one and then wait
    // for this one to be used
    const unsigned part = n_win / kFieldMakers;
    if (have == part) made_wait((int)((part + 1) & 1u));
    if (tt == 0) {
      end.words = (unsigned long long)kWin * n_win + (unsigned long long)o;
      end.done = 1;
    }
    __syncwarp();
    used_arrive((int)(part & 1u));
    if (who == 2 && lane == 0) {
      J.counters[kCntExpFp64] += st.fp64;
      J.counters[kCntExpCr] += st.cr;
    }
    if (who == 3 && lane == 0) {
      W.e_out = e_ex;
      if (W.e_state) *W.e_state = e_ex;
      W.accepted = n_acc;
      unsigned long long* c = J.counters;
      c[kCntTrials] += (unsigned long long)W.n_trials;
      c[kCntEvaluated] += c_eval;
      c[kCntDraws] += (unsigned long long)n_base * (unsigned long long)W.n_trials + c_exp;
      c[kCntAccepted] += n_acc;
      c[kCntExpTests] += c_exp;
      c[kCntExactPath] += c_exact;
      if (status != kStatusOk) *J.status = status;
    }
  }
  __syncthreads();
  // ---- write back -----------------------------------------------------------
  for (int i = tid; i < nb; i += blockDim.x) {
    W.lng[start - 1 + i] = lng[i];
    W.hist[i] = hist[i];
    if (W.store) W.store_open[start - 1 + i] = sopen[i];
  }
  const uint32_t* src = reinterpret_cast<const uint32_t*>(smem + L.lat);
  uint32_t* dst = reinterpret_cast<uint32_t*>(J.lat);
  const int n4 = g.n_sites >> 2;
  for (int i = tid; i < n4; i += blockDim.x) dst[i] = ((src[i] >> 2) & 0x3f3f3f3fu) + 0x01010101u;
  for (int i = (n4 << 2) + tid; i < g.n_sites; i += blockDim.x) J.lat[i] = (int8_t)((smem[L.lat + i] >> 2) + 1);
  if (tid == 0 && J.t_ns) *J.t_ns = global_ns() - t_start;
}

template <int NJ, int R>
static void launch_wl_field_r(WlWalker* d_walkers, int n, uint32_t smem, int threads, cudaStream_t stream) {
  BRAWL_SHARED(kWlFieldOwn, wl_field_kernel<NJ, R>);
  wl_field_kernel<NJ, R><<<n, threads, smem, stream>>>(d_walkers);
}

template <int NJ>
static void launch_wl_field_nj(WlWalker* d_walkers, int n, uint32_t smem, int variant, int threads,
                               cudaStream_t stream) {
  switch (variant) {
    case 1: launch_wl_field_r<NJ, 1>(d_walkers, n, smem, threads, stream); break;
    case 2: launch_wl_field_r<NJ, 2>(d_walkers, n, smem, threads, stream); break;
    case 4: launch_wl_field_r<NJ, 4>(d_walkers, n, smem, threads, stream); break;
    default: launch_wl_field_r<NJ, 0>(d_walkers, n, smem, threads, stream); break;
  }
}

// Walkers of one field_variant, neighbour counts up to max_z.
void launch_wl_field(WlWalker* d_walkers, int n, uint32_t smem, int max_z, int variant, cudaStream_t stream) {
  if (n <= 0) return;
  const int threads = 256;  // the roles' eight warps (more would leave them too few registers)
  if (max_z <= kFieldHalf) launch_wl_field_nj<1>(d_walkers, n, smem, variant, threads, stream);
  else if (max_z <= 2 * kFieldHalf) launch_wl_field_nj<2>(d_walkers, n, smem, variant, threads, stream);
  else launch_wl_field_nj<3>(d_walkers, n, smem, variant, threads, stream);
}

template <int NJ>
static void preload_wl_field_nj(cudaFuncAttributes& a) {
  cudaFuncGetAttributes(&a, wl_field_kernel<NJ, 1>);
  cudaFuncGetAttributes(&a, wl_field_kernel<NJ, 2>);
  cudaFuncGetAttributes(&a, wl_field_kernel<NJ, 4>);
  cudaFuncGetAttributes(&a, wl_field_kernel<NJ, 0>);
}

void preload_wl_field_kernels() {
  cudaFuncAttributes a;
  preload_wl_field_nj<1>(a);
  preload_wl_field_nj<2>(a);
  preload_wl_field_nj<3>(a);
}

}  // namespace brawl
