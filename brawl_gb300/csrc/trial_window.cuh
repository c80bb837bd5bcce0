// trial_window.cuh -- a warp's look-ahead over its mt19937ar stream: the next
// stream positions, one per lane, each decoded as the trial that would start
// there.
//
// A trial starts at the word after the previous trial's last one, and a trial
// draws a word more when it goes uphill, so where the next ones start is only
// known one after the other.  What a trial needs that does not depend on the
// energies -- its two sites and their species -- is decoded for 32 positions
// (a window) at once, by the lanes.  About five trials start in a window, so
// one warp-wide decode serves five trials, where decoding per trial has all
// 32 lanes do the same work.
//
// Stream.  The words are kept untempered in a ring of kMtRing, regenerated 32
// at a time ahead of the windows (word s needs words s - 624, s - 623 and
// s - 227), and tempered into a second ring.  The first ring holds the whole
// block the stream stands in whatever was generated ahead, so the state is
// put back in the reference's form (mt[624], mti) by copying it out.
#pragma once

#include "chain_engine.cuh"

namespace brawl {

constexpr int kWin = 32;              // positions per window
constexpr int kLookAhead = 3 * kWin;  // words generated before the first window
constexpr int kMtAhead = 6 * kWin;    // words generated ahead of the stream at most
constexpr int kMtRing = 26 * kWin;
constexpr int kMtMirror = kWin;       // the ring's first words again past its end
constexpr int kTwRing = 8 * kWin;     // tempered words held, again with
constexpr int kTwMirror = 8;          // the first ones past the end: a trial's words never wrap
static_assert(kMtRing >= kMTN + kMtAhead, "the block the stream stands in stays in the ring");
static_assert(kTwRing >= kMtAhead && kLookAhead + 2 * kWin <= kMtAhead, "the stream's words stay in the ring");

// Words of shared memory of the two rings.
constexpr int kRollWords = kMtRing + kMtMirror + kTwRing + kTwMirror;

struct MtRoll {
  int made;  // words up to here exist (from the start of the block as it was loaded), while < 624 + kWin
  int b;     // ring place of the next word once words are generated, a multiple of kWin plus pos0's
  int tg;    // its place in the ring of tempered words
};

// The block as it was loaded (words 0-623 of the stream's count) goes to ring
// places kMtRing - pos0 + word (modulo kMtRing), so that the word at the
// stream's position pos0, and every window after it, starts at a multiple of
// kWin.
__device__ __forceinline__ int mt_ring_place(int word, int pos0) {
  const int p = word - pos0;
  return p < 0 ? p + kMtRing : p;
}

__device__ __forceinline__ void mt_roll_load(const uint32_t* rng, uint32_t* mt, int pos0, int lane) {
  for (int i = lane; i < kMTN; i += 32) {
    const int p = mt_ring_place(i, pos0);
    const uint32_t v = rng[i];
    mt[p] = v;
    if (p < kMtMirror) mt[kMtRing + p] = v;
  }
}

// The next 32 words: into the ring (unless they are the loaded block's own)
// and tempered into tw.  Words s - 624, s - 623 and s - 227 sit that far back
// from place b, modulo the ring; a row of 32 that straddles the ring's end
// reads on into the mirror.  The places read and written in one call
// are different ones: only a __syncwarp before the next call is needed.
__device__ __forceinline__ void mt_roll(uint32_t* mt, uint32_t* tw, MtRoll& R, int lane) {
  const int b = R.b;
  int b1 = b + (kMtRing - kMTN), b2 = b + (kMtRing - (kMTN - kMTM));
  b1 -= b1 >= kMtRing ? kMtRing : 0;
  b2 -= b2 >= kMtRing ? kMtRing : 0;
  uint32_t v = mt_mix(mt[b1 + lane], mt[b1 + 1 + lane], mt[b2 + lane]);
  if (R.made < kMTN) {  // (part of) the loaded block
    if (R.made + lane < kMTN) v = mt[b + lane];
  }
  if (R.made < kMTN + kWin) R.made += kWin;
  mt[b + lane] = v;
  if (b == 0) mt[kMtRing + lane] = v;
  const uint32_t t = mt_temper(v);
  tw[R.tg + lane] = t;
  if (R.tg == 0 && lane < kTwMirror) tw[kTwRing + lane] = t;
  R.b = b + kWin == kMtRing ? 0 : b + kWin;
  R.tg = R.tg + kWin == kTwRing ? 0 : R.tg + kWin;
}

// (mt, mti) in the reference's form after `used` words from position pos0 of
// the block as it was loaded, `made` words having been generated from there
// (used <= made <= used + kMtAhead).
__device__ inline void mt_roll_store(uint32_t* mt, uint32_t* tw, MtRoll& R, int pos0, unsigned long long used,
                                     unsigned long long made, uint32_t* out, int lane) {
  const unsigned long long next = (unsigned long long)pos0 + used;
  const unsigned long long blk = next <= kMTN ? 0ull : (next - 1) / kMTN;  // the block the last word is in
  const unsigned long long first = blk * kMTN;
  if (blk > 0)
    while ((unsigned long long)pos0 + made < first + kMTN) {
      __syncwarp();
      mt_roll(mt, tw, R, lane);
      made += kWin;
    }
  __syncwarp();
  // word s sits at place s - pos0 modulo the ring
  const int at = blk > 0 ? (int)((first - (unsigned long long)pos0) % kMtRing) : mt_ring_place(0, pos0);
  for (int i = lane; i < kMTN; i += 32) {
    const int p = at + i;
    out[i] = mt[p >= kMtRing ? p - kMtRing : p];
  }
  if (lane == 0) out[kMTN] = (uint32_t)(next - first);
}

// Positions whose records (see metropolis_halo.cu) are held: two windows.
constexpr int kRecRing = 2 * kWin;

// One site's entries padded to whole lane rows of 16, an odd number of them so
// that the two sites' tables start in different banks.
__host__ __device__ __forceinline__ int entry_pad(int z) { return 16 * (((z + 15) / 16) | 1); }

}  // namespace brawl
