// halo_engine.cuh -- the stream of the walker kernels, and the sites that fcc and
// bcc proposals draw.
//
// Stream.  mt19937ar words are consumed from a ring of two tempered blocks
// (tbuf); a block is generated (twist + temper) when the consumer gets
// within a trial of the end of the generated words, so a trial reads its
// words with plain shared loads.  The state written back is the reference's
// (mt[624], mti): when consumption is still in the older block, that block's
// untempered words are recovered by inverting the tempering.
#pragma once

#include "chain_engine.cuh"

namespace brawl {

// ---------------------------------------------------------------------------
// tempered ring
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t mt_untemper(uint32_t y) {
  // inverse of mt_temper, step by step from the last
  y ^= y >> 18;
  y ^= (y << 15) & 0xefc60000u;
  // y ^= (y << 7) & 0x9d2c5680: recover 7 bits at a time
  uint32_t t = y;
  t = y ^ ((t << 7) & 0x9d2c5680u);
  t = y ^ ((t << 7) & 0x9d2c5680u);
  t = y ^ ((t << 7) & 0x9d2c5680u);
  t = y ^ ((t << 7) & 0x9d2c5680u);
  y = t;
  // y ^= y >> 11
  t = y ^ (y >> 11);
  y = y ^ (t >> 11);
  return y;
}

// Ring of two tempered blocks in tbuf[0, 1248), plus a mirror of the first
// kRingMirror words at tbuf[1248, 1248 + kRingMirror) so the words of a
// trial (or of a batch of redraws) never wrap.  `idx` is the
// ring slot of the next word, `avail` the generated words not yet consumed
// (0..1248), `next_half` the half the next generated block goes to; mt holds
// the newest generated block, untempered.
constexpr int kRing = 2 * kMTN;

struct Ring {
  int idx;
  int avail;
  int next_half;
};

// Twists mt in place and tempers the new block into the ring half next_half.
static __device__ __noinline__ void ring_generate(uint32_t* mt, uint32_t* tbuf, int next_half,
                                           int lane) {
  mt_twist_warp(mt, lane);
  uint32_t* dst = tbuf + next_half * kMTN;
  for (int i = lane; i < kMTN; i += 32) dst[i] = mt_temper(mt[i]);
  if (next_half == 0)
    for (int i = lane; i < kRingMirror; i += 32) tbuf[kRing + i] = mt_temper(mt[i]);
  __syncwarp();
}

// The block in mt is current with mti = pos0 (0..624): temper it into half 0.
__device__ __forceinline__ void ring_init(const uint32_t* mt, uint32_t* tbuf, int pos0, int lane,
                                          Ring& R) {
  for (int i = lane; i < kMTN; i += 32) tbuf[i] = mt_temper(mt[i]);
  for (int i = lane; i < kRingMirror; i += 32) tbuf[kRing + i] = mt_temper(mt[i]);
  R.idx = pos0;
  R.avail = kMTN - pos0;
  R.next_half = 1;
  __syncwarp();
}

// Makes n <= kRingMirror words available from R.idx.  A block is only generated when
// fewer than n remain, so the half it overwrites has been consumed.
__device__ __forceinline__ void ring_ensure(uint32_t* mt, uint32_t* tbuf, Ring& R, int n,
                                            int lane) {
  if (R.avail < n) {
    ring_generate(mt, tbuf, R.next_half, lane);
    R.avail += kMTN;
    R.next_half ^= 1;
  }
}

__device__ __forceinline__ void ring_consume(Ring& R, int n) {
  R.idx += n;
  R.idx = R.idx >= kRing ? R.idx - kRing : R.idx;
  R.avail -= n;
}

// Writes (mt, mti) in the reference's form.  If the next word lies in the
// block before the newest one, that block is recovered by untempering.
__device__ inline void ring_writeback(const uint32_t* mt, const uint32_t* tbuf, const Ring& R,
                                      uint32_t* out, int lane) {
  if (R.avail <= kMTN) {
    for (int i = lane; i < kMTN; i += 32) out[i] = mt[i];
    if (lane == 0) out[kMTN] = (uint32_t)(kMTN - R.avail);
  } else {
    const int older = R.next_half;  // the half after the newest is the older one
    for (int i = lane; i < kMTN; i += 32) out[i] = mt_untemper(tbuf[older * kMTN + i]);
    if (lane == 0) out[kMTN] = (uint32_t)(kRing - R.avail);
  }
}

// draw_site for fcc and bcc, also giving the site's compact (Y', X') =
// (y >> ys, x >> 1) without going through the doubled coordinates.
__device__ __forceinline__ void draw_site_halo(const Geom& g, bool bcc, uint32_t w0, uint32_t w1,
                                               uint32_t w2, int& x, int& y, int& z, int& Yc,
                                               int& Xc) {
  z = (int)umulhi32(w0, 2u * g.n3);
  if (bcc) {
    const int p = z & 1;
    Xc = (int)umulhi32(w1, (uint32_t)g.n1);
    Yc = (int)umulhi32(w2, (uint32_t)g.n2);
    x = 2 * Xc + p;
    y = 2 * Yc + p;
  } else {
    x = (int)umulhi32(w1, 2u * g.n1);
    y = 2 * (int)umulhi32(w2, (uint32_t)g.n2) + ((x + z) & 1);
    Yc = y;
    Xc = x >> 1;
  }
}

}  // namespace brawl
