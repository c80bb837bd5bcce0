// trial_window.cuh -- a warp's look-ahead over its mt19937ar stream: the next
// 32 stream positions, one per lane, each decoded as the trial that would
// start there.
//
// A trial starts at the word after the previous trial's last one, and a trial
// draws a word more when it goes uphill, so where the next ones start is only
// known one after the other.  What a trial needs that does not depend on the
// energies -- its two sites, their species, its acceptance thresholds -- is
// decoded for every position at once, 32 at a time, by the lanes; a trial
// then takes its position's values with shuffles.  About five trials start in
// a window of 32 words, so one warp-wide decode serves five trials, where
// decoding per trial has all 32 lanes do the same work.
//
// Stream.  The 624-word block is regenerated in place 32 words at a time
// (word k of the next block needs words k, k + 1 and k + 397 of the running
// sequence, all older than the batch), always kLookAhead words ahead of the
// window's start, and the tempered words pass through a ring of 128.  At the
// end the block is put back in the reference's form (mt[624], mti): the first
// words of a block that was begun ahead of the stream are kept in `old`.
#pragma once

#include "chain_engine.cuh"

namespace brawl {

constexpr int kWin = 32;           // positions per window
constexpr int kTwRing = 128;       // tempered words held
constexpr int kTwMirror = 8;       // the ring's first words again past its end: a trial's words never wrap
constexpr int kLookAhead = 3 * kWin;  // words generated past the next window's start
constexpr int kOldWords = 128;     // overwritten words kept per block: at most kLookAhead + kWin

// Words of shared memory: the block, the kept words, the tempered ring.
constexpr int kRollWords = kMTN + kOldWords + kTwRing + kTwMirror;

struct MtRoll {
  int kg;       // block slot of the next word to generate (624: the next block's first)
  int tg;       // its place in the ring, a multiple of 32
  bool fresh;   // slots from kg on hold the previous block (false: the block as it was loaded)
};

// The next 32 words into the ring, regenerating their slots (or, in the block
// as it was loaded, just tempering them).
__device__ __forceinline__ void mt_roll(uint32_t* mt, uint32_t* old, uint32_t* tw, MtRoll& R, int lane) {
  int k = R.kg + lane;
  const bool wrap = k >= kMTN;
  k -= wrap ? kMTN : 0;
  const bool fresh = R.fresh || wrap;
  const int k1 = k + 1 == kMTN ? 0 : k + 1;
  const int km = k + kMTM >= kMTN ? k + kMTM - kMTN : k + kMTM;
  const uint32_t x = mt[k];
  const uint32_t y = mt_mix(x, mt[k1], mt[km]);
  const uint32_t v = fresh ? y : x;
  __syncwarp();
  if (fresh) {
    if (k < kOldWords) old[k] = x;
    mt[k] = v;
  }
  const uint32_t t = mt_temper(v);
  tw[R.tg + lane] = t;
  if (R.tg == 0 && lane < kTwMirror) tw[kTwRing + lane] = t;
  __syncwarp();
  R.kg += kWin;
  if (R.kg >= kMTN) {
    R.kg -= kMTN;
    R.fresh = true;
  }
  R.tg = (R.tg + kWin) & (kTwRing - 1);
}

// (mt, mti) in the reference's form after `used` words from position pos0 of
// the block as it was loaded, `made` words having been generated from there
// (made >= used, made - used <= kOldWords).
__device__ inline void mt_roll_store(uint32_t* mt, uint32_t* old, uint32_t* tw, MtRoll& R, int pos0,
                                     unsigned long long used, unsigned long long made, uint32_t* out,
                                     int lane) {
  const unsigned long long next = (unsigned long long)pos0 + used;
  const unsigned long long blk = next <= kMTN ? 0ull : (next - 1) / kMTN;  // the block the last word is in
  const unsigned long long end = (blk + 1) * kMTN;
  unsigned long long gen = (unsigned long long)pos0 + made;
  if (blk > 0)
    while (gen < end) {
      mt_roll(mt, old, tw, R, lane);
      gen += kWin;
    }
  const int r = gen > end ? (int)(gen - end) : 0;  // slots already in the block after it
  for (int i = lane; i < kMTN; i += 32) out[i] = i < r ? old[i] : mt[i];
  if (lane == 0) out[kMTN] = (uint32_t)(next - blk * kMTN);
}

}  // namespace brawl
