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

constexpr int kWin = 32;      // positions per window
constexpr int kMtMirror = kWin;  // the word ring's first words again past its end
constexpr int kTwMirror = 8;     // and the tempered ring's: a trial's words never wrap

// The two rings of a kernel that generates up to Ahead words (a multiple of
// kWin) ahead of the stream: the words, the whole block the stream stands in
// among them, and the tempered words.
template <int Ahead>
struct StreamRing {
  static constexpr int kMt = (kMTN + Ahead + kWin - 1) / kWin * kWin;
  static constexpr int kTw = Ahead;
  static constexpr int kTwAt = kMt + kMtMirror;  // the tempered ring's place after the words
  static constexpr int kWords = kTwAt + kTw + kTwMirror;
};

struct MtRoll {
  int made;  // words up to here exist (from the start of the block as it was loaded), while < 624 + kWin
  int b;     // ring place of the next word, a multiple of kWin
  int tg;    // its place in the ring of tempered words
};

// Word s of the stream's count (0-623: the block as it was loaded) goes to ring
// place s - pos0 modulo the ring, so that the word at the stream's position pos0,
// and every window after it, starts at a multiple of kWin.
template <class Ring>
__device__ __forceinline__ void mt_roll_load(const uint32_t* rng, uint32_t* mt, int pos0, int lane) {
  for (int i = lane; i < kMTN; i += 32) {
    const int p = i < pos0 ? i - pos0 + Ring::kMt : i - pos0;
    const uint32_t v = rng[i];
    mt[p] = v;
    if (p < kMtMirror) mt[Ring::kMt + p] = v;
  }
}

// The next 32 words: into the ring (unless they are the loaded block's own) and
// tempered into tw; then `skip` more rows belong to other warps.  Words s - 624,
// s - 623 and s - 227 sit that far back from place b, modulo the ring; a row of
// 32 that straddles the ring's end reads on into the mirror.  The places read
// and written in one call (and in a row of calls up to 195 words apart) are
// different ones.
template <class Ring>
__device__ __forceinline__ void mt_roll(uint32_t* mt, uint32_t* tw, MtRoll& R, int lane, int skip = 0) {
  const int b = R.b;
  const int b1 = b >= kMTN ? b - kMTN : b - kMTN + Ring::kMt;
  const int b2 = b >= kMTN - kMTM ? b - (kMTN - kMTM) : b - (kMTN - kMTM) + Ring::kMt;
  uint32_t v = mt_mix(mt[b1 + lane], mt[b1 + 1 + lane], mt[b2 + lane]);
  if (R.made < kMTN) {  // (part of) the loaded block
    if (R.made + lane < kMTN) v = mt[b + lane];
  }
  if (R.made < kMTN + kWin) R.made += (1 + skip) * kWin;
  mt[b + lane] = v;
  if (b == 0) mt[Ring::kMt + lane] = v;
  const uint32_t t = mt_temper(v);
  tw[R.tg + lane] = t;
  if (R.tg == 0 && lane < kTwMirror) tw[Ring::kTw + lane] = t;
  const int nb = b + (1 + skip) * kWin, nt = R.tg + (1 + skip) * kWin;
  R.b = nb >= Ring::kMt ? nb - Ring::kMt : nb;
  R.tg = nt >= Ring::kTw ? nt - Ring::kTw : nt;
}

// (mt, mti) in the reference's form after `used` words from position pos0 of
// the block as it was loaded, `made` words having been generated from there
// (used <= made <= used + the ring's Ahead).  R: the next row's.
template <class Ring>
__device__ inline void mt_roll_store(uint32_t* mt, uint32_t* tw, MtRoll& R, int pos0, unsigned long long used,
                                     unsigned long long made, uint32_t* out, int lane) {
  const unsigned long long next = (unsigned long long)pos0 + used;
  const unsigned long long blk = next <= kMTN ? 0ull : (next - 1) / kMTN;  // the block the last word is in
  const unsigned long long first = blk * kMTN;
  if (blk > 0)
    while ((unsigned long long)pos0 + made < first + kMTN) {
      __syncwarp();
      mt_roll<Ring>(mt, tw, R, lane);
      made += kWin;
    }
  __syncwarp();
  // word s sits at place s - pos0 modulo the ring
  const int at = blk > 0 ? (int)((first - (unsigned long long)pos0) % Ring::kMt) : (pos0 > 0 ? Ring::kMt - pos0 : 0);
  for (int i = lane; i < kMTN; i += 32) {
    const int p = at + i;
    out[i] = mt[p >= Ring::kMt ? p - Ring::kMt : p];
  }
  if (lane == 0) out[kMTN] = (uint32_t)(next - first);
}

// Whether the sites drawn by words w[0..2] and w[3..5] may lie within given
// offsets of each other, from the words alone (never false for two that do; the
// host's words_within makes the constants and has the margin).
__device__ __forceinline__ bool words_near(const uint32_t c[3], const uint32_t c2[3], const uint32_t* w) {
  return (w[3] - w[0] + c[0] <= c2[0]) & (w[4] - w[1] + c[1] <= c2[1]) & (w[5] - w[2] + c[2] <= c2[2]);
}

// The gather kernel's (metropolis_halo.cu): words generated before the first
// window, the rings, and the positions whose records are held.
constexpr int kLookAhead = 3 * kWin;
using GatherRing = StreamRing<kLookAhead + 3 * kWin>;
constexpr int kRecRing = 2 * kWin;

// One site's entries padded to whole lane rows of 16, an odd number of them so
// that the two sites' tables start in different banks.
__host__ __device__ __forceinline__ int entry_pad(int z) { return 16 * (((z + 15) / 16) | 1); }

}  // namespace brawl
