// metropolis_field.cu -- Metropolis-Kawasaki swap trials for fcc/bcc chains
// whose sites' fields fit in shared memory (field_engine.cuh); trials in the
// reference's order (monte_carlo_step_lattice / _nbr,
// src/metropolis.F90:751-891) on the chain's own mt19937ar stream.
#include <algorithm>
#include <functional>

#include "accept_thresholds.cuh"
#include "field_engine.cuh"

namespace brawl {

// What the team shares of two windows (twice: one pair is written while the
// other is read): the walk from every position, each position's change and
// species (as stored, site 2's from bit 8), and the masks of rejections.
struct FieldShare {
  unsigned walk[2][2 * kWin];
  int2 pos[2][2 * kWin];
  unsigned rej[2][2];
  int verdict;  // the exact tier's: bit 0 accepted, bit 1 uniform drawn
};
static_assert(own_bytes<FieldEnd, FieldShare>() == kFieldOwn, "what the layout leaves room for");

// One chain per block.  All warps stage the tables and sum the fields; then four
// make the windows' records and the team of four decides the trials.  The team
// goes in step: two of its warps decide a window each (32 positions, one per
// lane, on the lattice as it stands) and walk through it from every position; all
// four then follow the walk to the first trial that is not certainly rejected,
// and update the fields together when it is accepted.
//
// What bounds it: the chain's dependent sequence times the longest chain's
// trials.  A pair of windows (nine or ten trials) costs the latency of two
// dependent shared loads, a ballot, a barrier and the walk; an accepted trial
// that of an update shared by 128 threads.  On one chain the other schedulers
// of the SM are idle, so the team's repeated work costs nothing.
template <int NJ, int R>
__global__ void __launch_bounds__(512, 1) metropolis_field_kernel(const ChainJob* __restrict__ jobs) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ FieldEnd end;
  __shared__ __align__(16) FieldShare S;
  const ChainJob& J = jobs[blockIdx.x];
  if (J.status && *J.status != 0) return;  // the chain's input was flagged: no trial runs
  const Geom g = J.g;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned long long t_start = global_ns();
  const FieldLayout L = field_layout(g, J.fg);
  if (tid == 0) end.done = 0;
  field_stage(J, g, L, smem, tid, blockDim.x);
  // Warps 2, 3, 6 and 7 are the team (the schedulers take every fourth warp, so
  // it has two of them to itself), 0, 1, 4 and 5 the makers.
  if (warp < 8 && (warp & 2) == 0) {
    // A's last word: the larger of rej_above and the band; B's third: acc_below
    const int band = J.band;
    const float inv_k = 1.0f / J.beta_q_l2, band_f = (float)band;
    field_produce(J, g, L, smem, &end, (warp & 1) + (warp >> 1), lane, [=](uint32_t w) {
      const AcceptThresholds th = accept_thresholds(w, inv_k, band_f);
      return make_int2(max(band, th.rej_above), th.acc_below);
    });
  } else if (warp < 8) {
    const int who = (warp & 1) + (warp >> 2) * 2, tt = who * 32 + lane;
    const bool second = tt >= kFieldHalf;
    FieldPlan<NJ> P;
    field_plan<NJ>(g, L, smem, tt, P);
    const int distinct = J.fg.distinct;
    const bool nbr = J.nbr_swap != 0;
    const int n_base = nbr ? 4 : 6;
    const int nt = (int)J.n_trials;
    const int band = J.band, ns = g.ns, r = field_stride(ns), stride = 4 * r, per = g.nsh * stride;
    // 32-bit tallies (a launch runs fewer than 2^31 trials per chain); the
    // uniforms follow from the words consumed
    unsigned b_like = 0, b_rej = 0, b_event = 0, b_acc = 0, b_exact = 0, c_fp64 = 0, c_cr = 0;
    unsigned n_win = 0;      // windows passed
    int o = 0, t = 0;        // the next trial's position in the window; trials done
    int slot = 0;            // the window's place in the record ring
    unsigned have = 0;       // the last part waited for
    int flip = 0;            // the shared pair in use
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
    while (t < nt) {
      if (who < 2) {
        const int4 a = *reinterpret_cast<const int4*>(smem + FieldLayout::kA + (after(slot, kWin * who) + lane) * 16);
        const int sa = smem[L.lat + a.x], sb = smem[L.lat + a.y];
        // species 1 (0 as stored) has no field: its loads are read past
        const unsigned char* ga = smem + L.g - 4 + a.x * stride;
        const unsigned char* gb = smem + L.g - 4 + a.y * stride;
        const int ab = *reinterpret_cast<const int32_t*>(ga + sb), bb = *reinterpret_cast<const int32_t*>(gb + sb);
        const int ba = *reinterpret_cast<const int32_t*>(gb + sa), aa = *reinterpret_cast<const int32_t*>(ga + sa);
        const int met = *reinterpret_cast<const int32_t*>(smem + a.z + sa * ns + sb);
        const int dE = (sb ? ab - bb : 0) + (sa ? ba - aa : 0) + met;
        // (rej_above >= acc_below: a trial above rej_above is not also below it)
        const unsigned like = __ballot_sync(kFull, sa == sb);
        const unsigned rej = __ballot_sync(kFull, sa != sb && dE > a.w);
        S.pos[flip][tt] = make_int2(dE, sa | sb << 8);
        S.walk[flip][tt] = field_walk(like, rej, lane, n_base, nbr);
        if (lane == 0) S.rej[flip][who] = rej;
      }
      team_sync();
      const unsigned w0 = S.walk[flip][o];
      const int o0 = (int)(w0 & 0xffu);
      const unsigned w1 = o0 >= kWin ? S.walk[flip][o0] : 0u;
      const unsigned w = w0 + w1;  // (the counts; the positions apart)
      const int passed = (int)((w >> 8) & 0xffu), n_rej = (int)(w >> 16);
      if (passed >= nt - t) {
        // the run ends among the passed trials
        int k = 0;
        for (; t < nt; ++t) {
          const unsigned re = (S.rej[flip][k] >> o) & 1u;
          b_like += 1u - re;
          b_rej += re;
          o += n_base + (int)re;
          if (o >= kWin) {
            o -= kWin;
            ++k;
          }
        }
        pass_windows(k);
        break;
      }
      t += passed;
      b_rej += n_rej;
      b_like += passed - n_rej;
      const int e = o0 >= kWin;
      const int p = e ? (int)(w1 & 0xffu) : o0;
      if (p >= kWin) {
        flip ^= 1;
        o = p - kWin;
        pass_windows(2);
        continue;
      }
      // ---- a trial that is not certainly rejected ---------------------------
      const int at = after(slot, kWin * e) + p;
      const int4 a = *reinterpret_cast<const int4*>(smem + FieldLayout::kA + at * 16);
      const int4 q = *reinterpret_cast<const int4*>(smem + FieldLayout::kB + at * 16);
      const int2 v = S.pos[flip][kWin * e + p];
      const int s1 = v.y & 0xff, s2 = v.y >> 8;
      ++t;
      ++b_event;
      o = p + n_base + (v.x > band);
      int accept = v.x < -band || (v.x > band && v.x < q.z) ? 1 : -1;
      if (accept < 0) {
        // inside the band, or too near its threshold: the reference's FP64
        // sums, in its order
        ++b_exact;
        if (who == 0) {
          const double2 pair = field_exact_pair(field_exact_setup(g, L), q.x, q.y, a.x, a.y, (s1 >> 2) + 1,
                                                (s2 >> 2) + 1, lane);
          const double delta_e = __dsub_rn(pair.y, pair.x);
          int verdict = 1;
          if (!(delta_e < 0.0)) {
            DecideStats st = {0u, 0u};
            const uint32_t* tw = reinterpret_cast<const uint32_t*>(smem) + FieldWords::kTwAt;
            const uint32_t wu = tw[((n_win + e) % (FieldWords::kTw / kWin)) * kWin + p + n_base];
            verdict = u_lt_exp(wu, __dmul_rn(-J.beta, delta_e), st) | 2;
            c_fp64 += st.fp64;
            c_cr += st.cr;
          }
          if (lane == 0) S.verdict = verdict;
        }
        team_sync();
        const int verdict = *(volatile int*)&S.verdict;
        accept = verdict & 1;
        o = p + n_base + (verdict >> 1);
      }
      if (accept) {
        ++b_acc;
        if (tt == 0) {
          smem[L.lat + a.x] = (unsigned char)s2;
          smem[L.lat + a.y] = (unsigned char)s1;
        }
        // U's rows by (old - 1) ns + new - 1
        const int row = (int)L.U + ((second ? s2 * ns + s1 : s1 * ns + s2) >> 2) * per;
        int sites[NJ];
        field_sites<NJ>(smem, P, second ? q.y : q.x, sites);
        field_update<NJ, R>(L, smem, P, distinct, r, sites, row, q.w != 0, second);
      }
      pass_windows(e + (o >= kWin));
      o &= kWin - 1;
      team_sync();
    }
    // the makers have made, or are making, the part after this one and then wait
    // for this one to be used
    const unsigned part = n_win / kFieldMakers;
    if (have == part) made_wait((int)((part + 1) & 1u));
    const unsigned long long words = (unsigned long long)kWin * n_win + (unsigned long long)o;
    if (tt == 0) {
      end.words = words;
      end.done = 1;
    }
    __syncwarp();
    used_arrive((int)(part & 1u));
    if (tt == 0) {
      unsigned long long* c = J.counters;
      c[kCntTrials] += (unsigned long long)nt;
      c[kCntEvaluated] += b_rej + b_event;
      c[kCntDraws] += words;
      c[kCntAccepted] += b_like + b_acc;
      c[kCntExpTests] += words - (unsigned long long)n_base * (unsigned long long)nt;
      c[kCntExactPath] += b_exact;
      c[kCntExpFp64] += c_fp64;
      c[kCntExpCr] += c_cr;
    }
  }
  __syncthreads();
  // ---- write back -----------------------------------------------------------
  const uint32_t* src = reinterpret_cast<const uint32_t*>(smem + L.lat);
  uint32_t* dst = reinterpret_cast<uint32_t*>(J.lat);
  const int n4 = g.n_sites >> 2;
  for (int i = tid; i < n4; i += blockDim.x) dst[i] = ((src[i] >> 2) & 0x3f3f3f3fu) + 0x01010101u;
  for (int i = (n4 << 2) + tid; i < g.n_sites; i += blockDim.x) J.lat[i] = (int8_t)((smem[L.lat + i] >> 2) + 1);
  if (tid == 0 && J.t_ns) *J.t_ns = global_ns() - t_start;
}

int field_threads(std::vector<int64_t>& trials, int n_sm) {
  const int n = (int)trials.size();
  if (n <= n_sm) return 512;
  std::sort(trials.begin(), trials.end(), std::greater<int64_t>());
  // when each SM is free, the earliest first; the next chain takes that one
  const auto later = std::greater<int64_t>();
  std::vector<int64_t> free_at(trials.begin(), trials.begin() + n_sm);
  std::make_heap(free_at.begin(), free_at.end(), later);
  for (int k = n_sm; k < n; ++k) {
    std::pop_heap(free_at.begin(), free_at.end(), later);
    free_at.back() += trials[k];
    if (8 * free_at.back() > 9 * trials[0]) return 256;
    std::push_heap(free_at.begin(), free_at.end(), later);
  }
  return 512;
}

template <int NJ, int R>
static void launch_field_r(const ChainJob* d_jobs, int n_jobs, int threads, uint32_t smem_bytes, cudaStream_t stream) {
  BRAWL_SHARED(kFieldOwn, metropolis_field_kernel<NJ, R>);
  metropolis_field_kernel<NJ, R><<<n_jobs, threads, smem_bytes, stream>>>(d_jobs);
}

template <int NJ>
static void launch_field_nj(const ChainJob* d_jobs, int n_jobs, int threads, uint32_t smem_bytes, int ns, cudaStream_t stream) {
  switch (field_variant(ns)) {
    case 1: launch_field_r<NJ, 1>(d_jobs, n_jobs, threads, smem_bytes, stream); break;
    case 2: launch_field_r<NJ, 2>(d_jobs, n_jobs, threads, smem_bytes, stream); break;
    case 4: launch_field_r<NJ, 4>(d_jobs, n_jobs, threads, smem_bytes, stream); break;
    default: launch_field_r<NJ, 0>(d_jobs, n_jobs, threads, smem_bytes, stream); break;
  }
}

// The chains are of ns's variant (field_variant), their neighbour counts up to
// max_z.
void launch_metropolis_field(const ChainJob* d_jobs, int n_jobs, int threads, uint32_t smem_bytes, int max_z, int ns,
                             cudaStream_t stream) {
  if (n_jobs <= 0) return;
  if (max_z <= kFieldHalf) launch_field_nj<1>(d_jobs, n_jobs, threads, smem_bytes, ns, stream);
  else if (max_z <= 2 * kFieldHalf) launch_field_nj<2>(d_jobs, n_jobs, threads, smem_bytes, ns, stream);
  else launch_field_nj<3>(d_jobs, n_jobs, threads, smem_bytes, ns, stream);
}

template <int NJ>
static void preload_field_nj(cudaFuncAttributes& a) {
  cudaFuncGetAttributes(&a, metropolis_field_kernel<NJ, 1>);
  cudaFuncGetAttributes(&a, metropolis_field_kernel<NJ, 2>);
  cudaFuncGetAttributes(&a, metropolis_field_kernel<NJ, 4>);
  cudaFuncGetAttributes(&a, metropolis_field_kernel<NJ, 0>);
}

void preload_field_kernels() {
  cudaFuncAttributes a;
  preload_field_nj<1>(a);
  preload_field_nj<2>(a);
  preload_field_nj<3>(a);
}

}  // namespace brawl
