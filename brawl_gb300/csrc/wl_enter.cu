// wl_enter.cu -- enter_energy_window (src/wang-landau.F90:643-741) of walkers
// whose sites' fields fit in shared memory (field_engine.cuh): what
// wang_landau.cu's wl_enter_kernel does, step for step, on the same state.
//
// The walk is biased so sharply towards the window's middle (sigma is a four-
// hundredth of the energy range) that a step is accepted when it leads there and
// rejected when it does not, nearly without exception, and a walk that has to
// climb out of the likely energies rejects most of its steps.  So the steps that
// start at each position of two windows of the stream are decided at once from
// the fields, in single precision with a bound on its error; like pairs and
// certain rejections are passed, and the first other step is taken on its own.
// Accepted moves are logged and their FP64 energies summed later
// (lazy_exact.cuh); a test that the bounds do not settle, or an energy that may
// lie in the window, takes the exact values.
#include <climits>

#include "field_engine.cuh"
#include "lazy_exact.cuh"
#include "wl_kernels.cuh"

namespace brawl {

namespace {

struct EnterLayout {
  uint32_t lazy, total;
};

__host__ __device__ inline EnterLayout enter_layout(const Geom& g, const FieldGeom& f, int cap) {
  EnterLayout L;
  L.lazy = field_layout(g, f).total;
  L.total = L.lazy + (cap > 0 ? lazy_bytes(g, cap) : 0);
  return L;
}

// What the team shares of two windows (twice, as in wl_field.cu), and what a
// walk leaves.
struct EnterShare {
  unsigned walk[2][2 * kWin];
  int2 pos[2][2 * kWin];  // the change; species as stored (site 2's from bit 8; bit 16: certainly accepted)
  double e_sw;
  int verdict;
  double e;  // the energy after the walk, its steps, and whether it is settled
  int t, status, ok;
};
static_assert(own_bytes<FieldEnd, EnterShare>() == kWlEnterOwn, "what the layout leaves room for");

// full_energy (src/bw_hamiltonian.f90:58-81): the site energies by all threads,
// their sum in site order on one, and the half.
__device__ double full_energy_block(const Geom& g, const int8_t* lat, const double* V, const uint32_t* ents,
                                    const int16_t* sstart, double* site_e, double* out, int tid, int nt) {
  for (int i = tid; i < g.n_sites; i += nt) {
    int x, y, z;
    decode_site(g, i, x, y, z);
    site_e[i] = site_energy_ref(g, lat, V, ents, sstart, x, y, z);
  }
  __syncthreads();
  if (tid == 0) {
    double e = 0.0;
#pragma unroll 8
    for (int i = 0; i < g.n_sites; ++i) e = __dadd_rn(e, site_e[i]);
    *out = __dmul_rn(0.5, e);
  }
  __syncthreads();
  const double e = *(volatile double*)out;
  __syncthreads();
  return e;
}

}  // namespace

uint32_t wl_enter_field_smem_bytes(const Geom& g, const FieldGeom& f, int cap) {
  return enter_layout(g, f, cap).total;
}

// The roles of metropolis_field_kernel.  A walk is one chain of dependent steps; the
// long ones, into windows far from the likely energies, reject nearly all of them,
// and a window of those takes some 700 cycles, where wl_enter_kernel takes 5,500 a
// step (the FP64 sums of both sites, one term after the other).  32 walkers of bcc
// 4^3, four species, six shells, into four windows: 19.4 ms with wl_enter_kernel,
// 1.2 ms here.
template <int NJ, int R>
__global__ void __launch_bounds__(256, 1) wl_enter_field_kernel(WlEnterJob* __restrict__ jobs) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ FieldEnd end;
  __shared__ __align__(16) EnterShare S;
  WlEnterJob& E = jobs[blockIdx.x];
  const ChainJob& J = E.job;
  const Geom g = J.g;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const FieldLayout L = field_layout(g, J.fg);
  const EnterLayout EL = enter_layout(g, J.fg, E.field_cap);
  const double* V = reinterpret_cast<const double*>(smem + FieldLayout::kV);
  const uint32_t* ents = reinterpret_cast<const uint32_t*>(smem + L.ents);
  const int16_t* sstart = reinterpret_cast<const int16_t*>(smem + L.sstart);
  const double target = __ddiv_rn(__dadd_rn(E.min_e, E.max_e), 2.0);
  const double cond = __dmul_rn(fabs(__dsub_rn(E.max_e, E.min_e)), 0.1);
  const double in_hi = __dsub_rn(E.max_e, cond), in_lo = __dadd_rn(E.min_e, cond);
  const int64_t reinit = (int64_t)g.n_sites * 250;
  // initial_setup on the walker's stream, by the first warp
  auto draw = [&]() {
    if (warp == 0) {
      uint32_t* mt = reinterpret_cast<uint32_t*>(smem);
      for (int i = lane; i < kMTN; i += 32) mt[i] = J.rng[i];
      int pos = (int)J.rng[kMTN];
      unsigned long long draws = 0;
      __syncwarp();
      const bool ok = initial_setup_warp(E.init, J.lat, mt, pos, draws, lane);
      __syncwarp();
      for (int i = lane; i < kMTN; i += 32) J.rng[i] = mt[i];
      if (lane == 0) {
        J.rng[kMTN] = (uint32_t)(pos < 0 ? 0 : pos);
        S.ok = ok;
      }
    }
    __syncthreads();
    return *(volatile int*)&S.ok != 0;
  };
  int status = kStatusOk;
  if (E.initial && !draw()) status = kStatusBadSpecies;
  __syncthreads();
  double e_un = 0.0;
  if (status == kStatusOk) {
    field_stage(J, g, L, smem, tid, blockDim.x);
    e_un = full_energy_block(g, J.lat, V, ents, sstart, E.site_e, &S.e, tid, blockDim.x);
  }
  int64_t steps = -1, i_steps = 0;
  bool staged = true;
  for (int64_t it = 1; it <= E.max_steps && status == kStatusOk; ++it) {
    if (++i_steps % reinit == 0) {
      i_steps = 0;
      if (!draw()) {
        status = kStatusBadSpecies;
        break;
      }
      staged = false;
    }
    if (e_un < in_hi && e_un > in_lo) {
      e_un = full_energy_block(g, J.lat, V, ents, sstart, E.site_e, &S.e, tid, blockDim.x);
      if (e_un < in_hi && e_un > in_lo) {
        steps = it;
        break;
      }
      continue;
    }
    if (!staged) field_stage(J, g, L, smem, tid, blockDim.x);
    staged = true;
    // ---- steps, up to the next redraw, the last one or an energy in the window --
    const int nt = (int)min(E.max_steps - it + 1, reinit - i_steps);
    if (tid == 0) end.done = 0;
    __syncthreads();
    if ((warp & 2) == 0) {
      // A's last word: log(u) as a float (within 1e-5 of it); B's third: the word
      field_produce(J, g, L, smem, &end, (warp & 1) + (warp >> 1), lane, [](uint32_t w) {
        float lw;
        asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(lw) : "f"(__uint2float_rn(w)));
        return make_int2(__float_as_int((lw - 32.0f) * 0.693147182f), (int)w);
      });
    } else {
      const int who = (warp & 1) + (warp >> 2) * 2, tt = who * 32 + lane;
      const bool second = tt >= kFieldHalf;
      // the entries are symmetric: the sites that have a swapped site as a
      // neighbour are its own neighbours
      FieldPlan<NJ> P;
      field_plan<NJ>(g, L, smem, tt, P, 1);
      const LazyLog LG = lazy_layout(g, smem + EL.lazy, E.field_cap);
      const int distinct = J.fg.distinct;
      const int n_base = 6;
      const int band = J.band, ns = g.ns, r = field_stride(ns), stride = 4 * r, per = g.nsh * stride, z = g.z;
      const int g_at = (int)L.g - 4;  // species 1 (0 as stored) has no field: its loads are read past
      const double sig2x2 = E.sig2x2;
      const double q1 = ldexp(1.0, -E.S);  // one fixed-point quantum
      // Energies in units of sqrt(sig2x2): d = a (2 b + a) for a change a from b
      // above the target.
      const double rs = __drcp_rn(__dsqrt_rn(sig2x2));
      const float qa = __double2float_rn(__dmul_rn(q1, rs));
      const bool scaled = qa > 1.0e-30f && qa < 1.0e30f;
      const float da = (float)(band + 2) * qa * (1.0f + 1.0e-6f);  // a's error, beside its roundings
      // e_ex: the exact energy before the n_log logged moves; after them it lies
      // in e_ex + [Dlo, Dhi] quanta
      double e_ex = e_un;
      long long Dlo = 0, Dhi = 0;
      int n_log = 0;
      int st_walk = kStatusOk;
      float b2 = 0.0f, db2 = 0.0f;  // 2 b at the interval's middle, twice its half width
      float e_mid = 0.0f;           // e_ex above the target, in those units
      bool lost = false;            // an update may round by more than a quantum: nothing is settled
      long long out_hi = 0, out_lo = 0;  // from out_hi quanta on, and down from out_lo, outside the window
      auto bounds = [&]() {
        const float lo = __ll2float_rn(Dlo) * qa, hi = __ll2float_rn(Dhi) * qa;
        b2 = 2.0f * e_mid + (lo + hi);
        // (the float of e_ex - target, of the ends and of their sums)
        db2 = ((hi - lo) + 4.0f * qa) * (1.0f + 1.0e-6f) + 1.0e-6f * (fabsf(e_mid) + fabsf(lo) + fabsf(hi));
      };
      auto rebase = [&]() {
        e_mid = __double2float_rn(__dmul_rn(__dsub_rn(e_ex, target), rs));
        lost = !scaled || quanta_bound(e_ex, E.S) >= (1ll << 51);
        const double hi = ldexp(__dsub_ru(in_hi, e_ex), E.S), lo = ldexp(__dsub_rd(in_lo, e_ex), E.S);
        out_hi = lost || !(hi < 1.0e17) ? LLONG_MAX : hi < -1.0e17 ? LLONG_MIN : (long long)ceil(hi);
        out_lo = lost || !(lo > -1.0e17) ? LLONG_MIN : lo > 1.0e17 ? LLONG_MAX : (long long)floor(lo);
        Dlo = Dhi = 0;
        bounds();
      };
      rebase();
      // log(u) < -d: certainly (1), certainly not (-1), or not settled (0), for a
      // change of dE quanta and log(u) within 1e-5 of lu.  The change's float, its
      // product with b and the sum are each within 1e-6 of |a| (|2 b| + |a|), the
      // reference's own squares within 1e-15 of (|2 b| + |a|)^2.
      auto test = [&](int dE, float lu) {
        const float a = (float)dE * qa;
        const float d = a * (b2 + a), size = fabsf(b2) + fabsf(a);
        const float m = 3.0e-5f + 2.0e-6f * (fabsf(a) * size + fabsf(lu)) + da * (size + fabsf(a) + da + db2) +
                        fabsf(a) * db2 + 1.0e-14f * size * size;
        const float s = d + lu;
        return lost ? 0 : (s < -m && lu > -100.0f) ? 1 : s > m ? -1 : 0;
      };
      DecideStats st = {0u, 0u};
      auto flush = [&]() {
        if (n_log == 0) return;
        lazy_sites_any<4>(g, V, sstart, LG, n_log, kFoldWangLandau, tt, kFieldTeam);
        team_sync();
        const double before = e_ex;
        e_ex = lazy_fold(LG, n_log, e_ex, kFoldWangLandau);
        if (!in_quanta(e_ex, before, Dlo, Dhi, q1)) st_walk = kStatusBandViolated;
        n_log = 0;
        rebase();
      };
      unsigned n_win = 0;  // windows passed
      int o = 0, t = 0;    // the next step's position in the window; steps done
      int slot = 0;        // the window's place in the record ring
      unsigned have = 0;   // the last part waited for
      int flip = 0;        // the shared pair in use
      bool inside = false;
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
      while (t < nt && !inside && st_walk == kStatusOk) {
        if (who < 2) {
          const int4 a = *reinterpret_cast<const int4*>(smem + FieldLayout::kA + (after(slot, kWin * who) + lane) * 16);
          const int sa = smem[L.lat + a.x], sb = smem[L.lat + a.y];
          const unsigned char* ga = smem + g_at + a.x * stride;
          const unsigned char* gb = smem + g_at + a.y * stride;
          const int ab = *reinterpret_cast<const int32_t*>(ga + sb), bb = *reinterpret_cast<const int32_t*>(gb + sb);
          const int ba = *reinterpret_cast<const int32_t*>(gb + sa), aa = *reinterpret_cast<const int32_t*>(ga + sa);
          const int met = *reinterpret_cast<const int32_t*>(smem + a.z + sa * ns + sb);
          const int dE = (sb ? ab - bb : 0) + (sa ? ba - aa : 0) + met;
          const int verdict = test(dE, __int_as_float(a.w));
          const unsigned like = __ballot_sync(kFull, sa == sb);
          const unsigned rej = __ballot_sync(kFull, sa != sb && verdict < 0);
          S.pos[flip][tt] = make_int2(dE, sa | sb << 8 | (verdict > 0 ? 1 << 16 : 0));
          S.walk[flip][tt] = field_walk(like, rej, lane, n_base, false);
        }
        team_sync();
        const unsigned w0 = S.walk[flip][o];
        const int o0 = (int)(w0 & 0xffu);
        const unsigned w1 = o0 >= kWin ? S.walk[flip][o0] : 0u;
        const int passed = (int)(((w0 + w1) >> 8) & 0xffu);
        if (passed >= nt - t) {
          // the run ends among the passed steps: stepped through one by one
          int k = 0;
          for (; t < nt; ++t) {
            const int2 v = S.pos[flip][o + kWin * k];
            o += n_base + ((v.y & 0xff) != ((v.y >> 8) & 0xff));
            if (o >= kWin) {
              o -= kWin;
              ++k;
            }
          }
          pass_windows(k);
          break;
        }
        t += passed;
        const int e = o0 >= kWin;
        const int p = e ? (int)(w1 & 0xffu) : o0;
        if (p >= kWin) {
          flip ^= 1;
          o = p - kWin;
          pass_windows(2);
          continue;
        }
        // ---- a step of its own -----------------------------------------------
        const int at = after(slot, kWin * e) + p;
        const int4 a = *reinterpret_cast<const int4*>(smem + FieldLayout::kA + at * 16);
        const int4 q = *reinterpret_cast<const int4*>(smem + FieldLayout::kB + at * 16);
        const int2 v = S.pos[flip][kWin * e + p];
        const int s1 = v.y & 0xff, s2 = (v.y >> 8) & 0xff;
        ++t;
        int verdict = (v.y >> 16) & 1;
        bool exact = false;
        double e_sw = 0.0;
        if (!verdict) {
          // the logged moves' exact energy may settle it
          flush();
          verdict = test(v.x, __int_as_float(a.w));
          if (verdict == 0) {
            exact = true;
            if (who == 0) {
              const double2 pr = field_exact_pair(field_exact_setup(g, L), q.x, q.y, a.x, a.y, (s1 >> 2) + 1,
                                                  (s2 >> 2) + 1, lane);
              // e_swapped = e_unswapped - pair_unswapped + pair_swapped
              const double es = __dadd_rn(__dsub_rn(e_ex, pr.x), pr.y);
              const double xa = __dsub_rn(es, target), xb = __dsub_rn(e_ex, target);
              const double d = __ddiv_rn(__dsub_rn(__dmul_rn(xa, xa), __dmul_rn(xb, xb)), sig2x2);
              const int yes = log_u_lt((uint32_t)q.z, -d, st);
              if (lane == 0) {
                S.e_sw = es;
                S.verdict = yes;
              }
            }
            team_sync();
            e_sw = *(volatile double*)&S.e_sw;
            verdict = *(volatile int*)&S.verdict;
          }
        }
        const int next_o = p + n_base + 1;
        if (verdict > 0) {
          int at_n[NJ];
          field_sites<NJ>(smem, P, second ? q.y : q.x, at_n);
          if (exact) {
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
            Dlo += (long long)v.x - band - 1;
            Dhi += (long long)v.x + band + 1;
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
        team_sync();
        if (verdict > 0) {
          if (Dlo < out_hi && Dhi > out_lo) {  // (outside otherwise)
            flush();
            inside = e_ex < in_hi && e_ex > in_lo;
          }
          if (n_log == LG.cap) flush();
        }
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
        S.e = e_ex;
        S.t = t;
        S.status = st_walk;
      }
      __syncwarp();
      used_arrive((int)(part & 1u));
    }
    __syncthreads();
    // ---- the walk's end: the lattice back, and on ---------------------------
    const uint32_t* src = reinterpret_cast<const uint32_t*>(smem + L.lat);
    uint32_t* dst = reinterpret_cast<uint32_t*>(J.lat);
    const int n4 = g.n_sites >> 2;
    for (int i = tid; i < n4; i += blockDim.x) dst[i] = ((src[i] >> 2) & 0x3f3f3f3fu) + 0x01010101u;
    for (int i = (n4 << 2) + tid; i < g.n_sites; i += blockDim.x) J.lat[i] = (int8_t)((smem[L.lat + i] >> 2) + 1);
    e_un = *(volatile double*)&S.e;
    const int t = *(volatile int*)&S.t;
    status = *(volatile int*)&S.status;
    it += t - 1;
    i_steps += t - 1;
    __syncthreads();
  }
  if (tid == 0) {
    E.steps = steps;
    E.energy = e_un;
    if (status != kStatusOk) *J.status = status;
  }
}

template <int NJ, int R>
static void launch_enter_r(WlEnterJob* d_jobs, int n, uint32_t smem, cudaStream_t stream) {
  BRAWL_SHARED(kWlEnterOwn, wl_enter_field_kernel<NJ, R>);
  wl_enter_field_kernel<NJ, R><<<n, 256, smem, stream>>>(d_jobs);
}

template <int NJ>
static void launch_enter_nj(WlEnterJob* d_jobs, int n, uint32_t smem, int variant, cudaStream_t stream) {
  switch (variant) {
    case 1: launch_enter_r<NJ, 1>(d_jobs, n, smem, stream); break;
    case 2: launch_enter_r<NJ, 2>(d_jobs, n, smem, stream); break;
    case 4: launch_enter_r<NJ, 4>(d_jobs, n, smem, stream); break;
    default: launch_enter_r<NJ, 0>(d_jobs, n, smem, stream); break;
  }
}

// Walkers of one field_variant, neighbour counts up to max_z.
void launch_wl_enter_field(WlEnterJob* d_jobs, int n, uint32_t smem, int max_z, int variant, cudaStream_t stream) {
  if (n <= 0) return;
  if (max_z <= kFieldHalf) launch_enter_nj<1>(d_jobs, n, smem, variant, stream);
  else if (max_z <= 2 * kFieldHalf) launch_enter_nj<2>(d_jobs, n, smem, variant, stream);
  else launch_enter_nj<3>(d_jobs, n, smem, variant, stream);
}

template <int NJ>
static void preload_enter_nj(cudaFuncAttributes& a) {
  cudaFuncGetAttributes(&a, wl_enter_field_kernel<NJ, 1>);
  cudaFuncGetAttributes(&a, wl_enter_field_kernel<NJ, 2>);
  cudaFuncGetAttributes(&a, wl_enter_field_kernel<NJ, 4>);
  cudaFuncGetAttributes(&a, wl_enter_field_kernel<NJ, 0>);
}

void preload_wl_enter_kernels() {
  cudaFuncAttributes a;
  preload_enter_nj<1>(a);
  preload_enter_nj<2>(a);
  preload_enter_nj<3>(a);
}

}  // namespace brawl
