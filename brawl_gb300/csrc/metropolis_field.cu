// metropolis_field.cu -- Metropolis-Kawasaki swap trials for fcc/bcc chains
// whose sites' fields fit in shared memory (field_engine.cuh); trials in the
// reference's order (monte_carlo_step_lattice / _nbr,
// src/metropolis.F90:751-891) on the chain's own mt19937ar stream.
#include "accept_thresholds.cuh"
#include "field_engine.cuh"
#include "halo_engine.cuh"

namespace brawl {

namespace {

// Named hardware barriers of the block's first two warps, per half h of the
// record ring: its records are made (1, 2); they have been used (3, 4).  The
// numbers are literals: a number in a register would reserve all sixteen.
__device__ __forceinline__ void made_arrive(int h) {
  if (h) asm volatile("bar.arrive 2, 64;" ::: "memory");
  else asm volatile("bar.arrive 1, 64;" ::: "memory");
}
__device__ __forceinline__ void made_wait(int h) {
  if (h) asm volatile("bar.sync 2, 64;" ::: "memory");
  else asm volatile("bar.sync 1, 64;" ::: "memory");
}
__device__ __forceinline__ void used_arrive(int h) {
  if (h) asm volatile("bar.arrive 4, 64;" ::: "memory");
  else asm volatile("bar.arrive 3, 64;" ::: "memory");
}
__device__ __forceinline__ void used_wait(int h) {
  if (h) asm volatile("bar.sync 4, 64;" ::: "memory");
  else asm volatile("bar.sync 3, 64;" ::: "memory");
}

// What the walking warp tells the stream's warp at the end.
struct FieldEnd {
  unsigned long long words;
  int done;
};

// Warp 1: the windows' static records, two windows ahead of warp 0 at most
// four.
__device__ __forceinline__ void field_produce(const ChainJob& J, const Geom& g, const FieldLayout& L,
                                              unsigned char* smem, FieldEnd* end, int lane) {
  uint32_t* mt = reinterpret_cast<uint32_t*>(smem);
  uint32_t* tw = mt + kMtRing + kMtMirror;
  const FieldGeom f = J.fg;
  const uint8_t* dtab = smem + L.dtab;
  const bool bcc = g.lattice == kBcc;
  const bool nbr = J.nbr_swap != 0;
  const int band = J.band;
  const float inv_k = 1.0f / J.beta_q_l2, band_f = (float)band;
  const int W1 = 2 * g.n1, W2 = 2 * g.n2, W3 = 2 * g.n3;
  const int pos0 = (int)J.rng[kMTN];
  mt_roll_load(J.rng, mt, pos0, lane);
  __syncwarp();
  MtRoll R = {pos0, 0, 0};
  mt_roll(mt, tw, R, lane);
  __syncwarp();
  mt_roll(mt, tw, R, lane);
  __syncwarp();
  unsigned long long made = 2 * kWin;
  int at = 0;  // the window's place in the ring of tempered words
  for (unsigned i = 0;; ++i) {
    const int h = (int)(i & 1u);
    if (i >= 2) used_wait(h);
    if (*(volatile int*)&end->done) break;
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {
      const uint32_t* w = tw + at + lane;
      int ax, ay, az, Ya, Xa, bx, by, bz, Yb, Xb;
      draw_site_halo(g, bcc, w[0], w[1], w[2], ax, ay, az, Ya, Xa);
      if (nbr) {
        // draw_nbr's neighbour; its steps are -1, 0, 1
        const int8_t* v = cNbrSwap[g.lattice][umulhi32(w[3], (uint32_t)g.nbr_k)];
        bx = wrap_fast(ax + v[0], W1);
        by = wrap_fast(ay + v[1], W2);
        bz = wrap_fast(az + v[2], W3);
        Yb = by >> g.ys;
        Xb = bx >> 1;
      } else {
        draw_site_halo(g, bcc, w[3], w[4], w[5], bx, by, bz, Yb, Xb);
      }
      const AcceptThresholds th = accept_thresholds(w[nbr ? 4 : 6], inv_k, band_f);
      const int t1 = wrap_fast(bx - ax + f.dm[0], W1), t2 = wrap_fast(by - ay + f.dm[1], W2),
                t3 = wrap_fast(bz - az + f.dm[2], W3);
      int cls = 0;
      if (t1 < f.side[0] && t2 < f.side[1] && t3 < f.side[2]) cls = dtab[(t3 * f.side[1] + t2) * f.side[0] + t1];
      const int ia = az * g.sz + Ya * g.sy + Xa, ib = bz * g.sz + Yb * g.sy + Xb;
      const int slot = (2 * h + k) * kWin + lane;
      *reinterpret_cast<int4*>(smem + FieldLayout::kAt + slot * 16) =
          make_int4(ax | ay << 10 | az << 20, bx | by << 10 | bz << 20, ia | ib << 16, cls);
      *reinterpret_cast<int2*>(smem + FieldLayout::kTh + slot * 8) = make_int2(max(band, th.rej_above), th.acc_below);
      mt_roll(mt, tw, R, lane);
      made += kWin;
      __syncwarp();
      at = at + kWin == kTwRing ? 0 : at + kWin;
    }
    made_arrive(h);
  }
  mt_roll_store(mt, tw, R, pos0, end->words, made, J.rng, lane);
}

}  // namespace

// One chain per block.  All warps stage the tables and sum the fields; then
// warp 1 makes the windows' records and warp 0 decides the trials.  What
// bounds it: the chain's dependent sequence -- per window of 32 positions two
// dependent shared loads (species, fields), two ballots and the stepping
// through the outcomes, per accepted trial the update of 2z sites' fields and
// the window again -- times the longest chain's trials.
template <int NJ>
__global__ void __launch_bounds__(256) metropolis_field_kernel(const ChainJob* __restrict__ jobs) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ FieldEnd end;
  const ChainJob& J = jobs[blockIdx.x];
  if (J.status && *J.status != 0) return;  // the chain's input was flagged: no trial runs
  const Geom g = J.g;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned long long t_start = global_ns();
  const FieldLayout L = field_layout(g, J.fg);
  if (tid == 0) end.done = 0;
  field_stage(J, g, L, smem, tid, blockDim.x);
  if (warp == 1) {
    field_produce(J, g, L, smem, &end, lane);
  } else if (warp == 0) {
    FieldPlan<NJ> P;
    field_plan<NJ>(g, L, smem, lane, P);
    const int n_base = J.nbr_swap ? 4 : 6;
    const int hops = J.nbr_swap ? 7 : 5;  // trials that start in a window, less one
    const int nt = (int)J.n_trials;
    const int band = J.band, ns = g.ns, n4 = 4 * g.n_sites;
    const uint32_t* tw = reinterpret_cast<const uint32_t*>(smem) + kMtRing + kMtMirror;
    // 32-bit tallies (a launch runs fewer than 2^31 trials per chain); the
    // uniforms follow from the words consumed
    unsigned b_eval = 0, b_acc = 0, b_exact = 0, c_fp64 = 0, c_cr = 0;
    const FieldExact X = field_exact_setup(g, L);
    unsigned n_win = 0;  // windows passed
    int o = 0, t = 0;    // the next trial's position in the window; trials done
    int4 at;             // this lane's position
    int2 th;
    unsigned like = 0, rej = 0;  // positions: two like species; certainly rejected
    int outcome = 0;             // sa | sb << 4 | certainly accepted << 8 | certainly downhill << 9
    auto window = [&]() {
      const int slot = (int)(n_win & 3u) * kWin + lane;
      at = *reinterpret_cast<const int4*>(smem + FieldLayout::kAt + slot * 16);
      th = *reinterpret_cast<const int2*>(smem + FieldLayout::kTh + slot * 8);
    };
    auto decide = [&]() {
      const int ia = at.z & 0xffff, ib = (int)((unsigned)at.z >> 16);
      const int sa = smem[L.lat + ia], sb = smem[L.lat + ib];
      const unsigned char* ga = smem + L.g + 4 * ia - 2 * n4;
      const unsigned char* gb = smem + L.g + 4 * ib - 2 * n4;
      int dE = 0;
      if (sb > 1) dE += *reinterpret_cast<const int32_t*>(ga + sb * n4) - *reinterpret_cast<const int32_t*>(gb + sb * n4);
      if (sa > 1) dE += *reinterpret_cast<const int32_t*>(gb + sa * n4) - *reinterpret_cast<const int32_t*>(ga + sa * n4);
      if (at.w) dE += *reinterpret_cast<const int32_t*>(smem + L.C + ((at.w * ns + sa - 1) * ns + sb - 1) * 4);
      const bool same = sa == sb;
      const bool down = dE < -band;
      const bool sure = down || (dE > band && dE < th.y);
      // (rej_above >= acc_below: a trial above rej_above is not also below it)
      like = __ballot_sync(kFull, same);
      rej = __ballot_sync(kFull, !same && dE > th.x);
      outcome = sa | sb << 4 | (sure ? 1 << 8 : 0) | (down ? 1 << 9 : 0);
    };
    made_wait(0);
    window();
    decide();
    while (t < nt) {
      if (o >= kWin) {
        o -= kWin;
        ++n_win;
        if ((n_win & 1u) == 0u) {
          const int h = (int)((n_win >> 1) & 1u);
          used_arrive(h ^ 1);
          made_wait(h);
        }
        window();
        decide();
      }
      // the positions the chain steps through from o: like pairs (accepted
      // without an energy evaluation or a draw) and certain rejections, up to
      // the first other trial or the window's end
      unsigned path = 1u << o;
      const unsigned pass = like | rej;
#pragma unroll
      for (int i = 0; i < 5; ++i) path |= ((path & like) << n_base) | ((path & rej) << (n_base + 1));
      if (hops > 5) {
        path |= ((path & like) << n_base) | ((path & rej) << (n_base + 1));
        path |= ((path & like) << n_base) | ((path & rej) << (n_base + 1));
      }
      const int passed = __popc(path & pass);
      if (passed >= nt - t) {
        // the run ends among them, at its last trial
        unsigned m = path & pass;
        for (int i = nt - t; i < passed; ++i) m &= ~(0x80000000u >> __clz(m));
        const int last = 31 - __clz(m);
        b_acc += __popc(m & like);
        b_eval += __popc(m & rej);
        o = last + n_base + (int)((rej >> last) & 1u);
        t = nt;
        break;
      }
      t += passed;
      b_acc += __popc(path & like);
      b_eval += __popc(path & rej);
      const unsigned stop = path & ~pass;
      if (stop == 0u) {
        const int last = 31 - __clz(path);
        o = last + n_base + (int)((rej >> last) & 1u);
        continue;
      }
      // ---- a trial that is not certainly rejected ---------------------------
      const int p = __ffs(stop) - 1;
      const int out = __shfl_sync(kFull, outcome, p);
      const int4 q = *reinterpret_cast<const int4*>(smem + FieldLayout::kAt + ((int)(n_win & 3u) * kWin + p) * 16);
      const int s1 = out & 15, s2 = (out >> 4) & 15;
      const int i1 = q.z & 0xffff, i2 = (int)((unsigned)q.z >> 16);
      ++t;
      ++b_eval;
      int accept = 1;
      if (out & (1 << 8)) {
        o = p + n_base + ((out >> 9) & 1 ? 0 : 1);
      } else {
        // inside the band, or too near its threshold: the reference's FP64
        // sums, in its order
        ++b_exact;
        const double delta_e = field_exact_delta(X, q.x, q.y, i1, i2, s1, s2, lane);
        o = p + n_base;
        if (!(delta_e < 0.0)) {
          DecideStats st = {0u, 0u};
          const uint32_t wu = tw[(int)(n_win & (kTwRing / kWin - 1)) * kWin + p + n_base];
          accept = u_lt_exp(wu, __dmul_rn(-J.beta, delta_e), st);
          ++o;
          c_fp64 += st.fp64;
          c_cr += st.cr;
        }
      }
      if (accept) {
        ++b_acc;
        field_swap<NJ>(g, L, smem, P, q.x, q.y, i1, i2, s1, s2, lane);
        __syncwarp();
        if (o < kWin) decide();
      }
    }
    const unsigned long long words = (unsigned long long)kWin * n_win + (unsigned long long)o;
    // the stream's warp: it has made, or is making, the half after this one and
    // then waits for this one to be used
    const int h = (int)((n_win >> 1) & 1u);
    made_wait(h ^ 1);
    if (lane == 0) {
      end.words = words;
      end.done = 1;
    }
    __syncwarp();
    used_arrive(h);
    if (lane == 0) {
      unsigned long long* c = J.counters;
      c[kCntTrials] += (unsigned long long)nt;
      c[kCntEvaluated] += b_eval;
      c[kCntDraws] += words;
      c[kCntAccepted] += b_acc;
      c[kCntExpTests] += words - (unsigned long long)n_base * (unsigned long long)nt;
      c[kCntExactPath] += b_exact;
      c[kCntExpFp64] += c_fp64;
      c[kCntExpCr] += c_cr;
    }
  }
  __syncthreads();
  // ---- write back -----------------------------------------------------------
  const int8_t* lat = reinterpret_cast<const int8_t*>(smem + L.lat);
  const int n16 = g.n_sites >> 4;
  const uint4* src = reinterpret_cast<const uint4*>(lat);
  uint4* dst = reinterpret_cast<uint4*>(J.lat);
  for (int i = tid; i < n16; i += blockDim.x) dst[i] = src[i];
  for (int i = (n16 << 4) + tid; i < g.n_sites; i += blockDim.x) J.lat[i] = lat[i];
  if (tid == 0 && J.t_ns) *J.t_ns = global_ns() - t_start;
}

int field_threads(int n_sites) { return n_sites <= 512 ? 64 : n_sites <= 4096 ? 128 : 256; }

template <int NJ>
static void launch_field_nj(const ChainJob* d_jobs, int n_jobs, uint32_t smem_bytes, int threads, cudaStream_t stream) {
  cudaFuncSetAttribute(metropolis_field_kernel<NJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes);
  BRAWL_CARVEOUT(metropolis_field_kernel<NJ>);
  metropolis_field_kernel<NJ><<<n_jobs, threads, smem_bytes, stream>>>(d_jobs);
}

void launch_metropolis_field(const ChainJob* d_jobs, int n_jobs, uint32_t smem_bytes, int max_sites, int max_z,
                             cudaStream_t stream) {
  if (n_jobs <= 0) return;
  const int threads = field_threads(max_sites);
  switch (lane_entries_for(max_z)) {
    case 2: launch_field_nj<2>(d_jobs, n_jobs, smem_bytes, threads, stream); break;
    case 4: launch_field_nj<4>(d_jobs, n_jobs, smem_bytes, threads, stream); break;
    case 6: launch_field_nj<6>(d_jobs, n_jobs, smem_bytes, threads, stream); break;
    case 8: launch_field_nj<8>(d_jobs, n_jobs, smem_bytes, threads, stream); break;
    default: launch_field_nj<11>(d_jobs, n_jobs, smem_bytes, threads, stream); break;
  }
}

void preload_field_kernels() {
  cudaFuncAttributes a;
  cudaFuncGetAttributes(&a, metropolis_field_kernel<2>);
  cudaFuncGetAttributes(&a, metropolis_field_kernel<4>);
  cudaFuncGetAttributes(&a, metropolis_field_kernel<6>);
  cudaFuncGetAttributes(&a, metropolis_field_kernel<8>);
  cudaFuncGetAttributes(&a, metropolis_field_kernel<11>);
}

}  // namespace brawl
