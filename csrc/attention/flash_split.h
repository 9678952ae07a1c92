// Which items the attention forward (flash_fwd.cu) works through: pairs of tiles of 128 queries, or single tiles whose keys its two softmax warpgroups
// share.
#pragma once
#include <math.h>

namespace llmctl {

// Whether single tiles are the better ones, for `heads` (sequences x heads) of `blocks` key blocks each.  Counted in steps of a CTA (a block for both
// warpgroups, 1.5 us at D = 128).  Pairs: the longest item and two steps around it, or the SMs' mean load; items that are more than the SMs go, the lightest,
// to the CTAs of the lightest, so they do not stand behind the longest (only without a mask, where all are equal).  Single tiles: half as long, and
// more of them: the second ones stand behind first ones of about the same length.  They read the keys twice as often, which the load
// of the SMs feels, with heads of 128 more than with heads of 64; hence the factors.  us, pairs / single tiles, rows that were read before and from HBM:
//   heads of 128: 16 x 22 blocks 41.2 / 37.7, 42.3 / 40.9; x 23 41.1 / 40.2, 42.2 / 43.6; 20 x 16 30.9 / 28.1, 32.2 / 30.9; x 17 31.6 / 30.7, 32.5 / 33.7;
//                 32 x 5 12.9 / 11.1, 13.8 / 12.2; x 7 16.2 / 15.3, 17.2 / 16.4; x 9 19.6 / 19.0, 20.6 / 20.4; x 10 22.9 / 22.7, 23.9 / 25.0;
//                 40 x 4 12.1 / 10.9, 13.0 / 12.1; x 5 12.5 / 13.1, 13.7 / 14.3; x 7 16.2 / 17.2, 17.2 / 18.7; 64 x 2 and 80 x 2: below
//   heads of 64:  12 x 32 51.3 / 45.2, 52.4 / 46.0; 16 x 24 39.6 / 36.8, 40.8 / 37.7; x 25 40.0 / 38.6, 40.9 / 39.4; 24 x 14 25.6 / 22.9, 26.6 / 23.8;
//                 48 x 4 10.6 / 9.0, 11.7 / 10.0; x 5 11.1 / 11.7, 11.8 / 12.3; 96 x 3 12.8 / 10.3, 13.7 / 11.2
// Where the two are within 4% of each other it may take either (heads of 128, 32 x 3: 8.6 / 8.7, 36 x 3: 8.4 / 8.7); a few sizes on whose
// far side single tiles would win stay pairs (96 x 3 above).
inline bool split_keys(int heads_, int blocks, int head_size, bool causal, int sms) {
  if (blocks < 2) return false;
  const double heads = heads_, half = ceil(blocks / 2.), odd = 2 * half - blocks;
  const double load = head_size == 128 ? 1.4 : 1.3;
  if (!causal) {
    const double pairs = ceil(heads * half / sms) * (blocks + 2.), single = heads * blocks / sms;
    return fmax(1.3 * ceil(single), load * single) * (half + 1.2) < pairs;
  }
  const double steps = half * (half + 1) - odd;
  const double pairs = fmax(blocks + 2., heads * (steps + 2 * half) / sms);
  const double second = heads * blocks > sms ? blocks - sms / heads_ + 1 + 2.4 : 0.;      // two items where the first ones are lightest
  const double single = fmax(1.3 * fmax(half + 1.2, second), load * heads * (steps - odd * (half - 1) + 1.2 * blocks) / sms);
  return single < pairs;
}

}  // namespace llmctl
