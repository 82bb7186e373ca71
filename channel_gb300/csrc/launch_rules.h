// The rules by which sizes choose a step's launch shapes.  None of them
// changes a result.  `nsm`: the device's SMs; `together`: how many times a
// handle's modes or pairs those of all handles that step together are (an
// ensemble's members share the GPU; 1 for a lone handle).
#pragma once

#include <cmath>

namespace chgpu {

// Solve form of a handle that has not been tuned: eight threads per pair
// while its blocks are one wave (16 pairs per 128-thread block, four blocks
// on each SM, 9728 pairs on 152; ms per mixed step against four threads per
// pair: 32x64x32 0.51 / 0.66, 47x96x47 1.07 / 1.28, 83x120x85 2.70 / 2.83, but
// 127x192x127 6.97 / 6.45), then four threads, then the fused kernel.  The line
// is the same in FP64 and double-float: eight threads per pair take 0.79 of the
// step of four at 1089 pairs, 0.96 at 7225, 0.99 at 9604, 1.06 at 12 321.
inline int default_solve_form(long long pairs, int nsm) { return pairs <= 16ll * 4 * nsm ? 5 : pairs < 65536 ? 3 : 1; }

// Eight threads per pair, blocks of 16 pairs: four parts (256 threads) where
// two blocks on each SM hold all of them, else two parts (128 threads).
inline bool solve_in_four_parts(int blocks, int nsm, double together) { return blocks * together <= 2.0 * nsm; }

// Rows per thread of k_rhs: the count that minimises the time of the fullest
// SM, three blocks at a time.  A block's time is its rows plus `start`, the four
// start-up rows of the windows (1 row's worth; 2 in the FP32 path, which waits
// on their loads); three resident blocks take 3 units a row, one or two take
// `one` and `two` (measured at 32x64x32 and 47x96x47: the FP64 pipe is nearly
// filled by one block, the FP32 path's latency is not).  Against a fixed 16:
// FP64 0.285 -> 0.157 ms a step at 32x64x32, 0.487 -> 0.382 at 47x96x47,
// 1.29 -> 1.06 at 79x101x75; mixed 0.138 -> 0.067, 0.184 -> 0.136, 0.35 -> 0.30.
// Over nine sizes from 16x40x16 to 127x64x127 and 20x250x240 the choice is within
// 8% of the best of 12 counts, at seven of them within 4%.
//
// Of the other handles of an ensemble one in eight counts: their steps run side
// by side, but not all in k_rhs at once.  ms per step with none, an eighth and
// all of them counted: 5 members FP64 1.486, 1.448, 1.517; 12 mixed 1.496,
// 1.451, 1.467; 24 mixed 2.959, 2.753, 2.703; 64 mixed 8.13, 7.51, 7.50, FP64
// 18.03, 17.09, 16.88.
struct RhsCost {
  int start;
  double one, two;
};
constexpr RhsCost kRhsCostFP64{1, 1.25, 2.1}, kRhsCostDD{1, 1.6, 2.4}, kRhsCostFP32{2, 1.95, 2.6};
constexpr int kRhsMaxRows = 32;
inline int rhs_rows(RhsCost c, int modes, int ny, int nsm, double together) {
  const double cols = (modes + 127) / 128 * (1.0 + (together - 1.0) / 8);
  int best = kRhsMaxRows;
  double cost = 1e300;
  for (int rb = kRhsMaxRows; rb >= 2; --rb) {
    const long long per_sm = (long long)std::ceil(cols * ((ny - 1 + rb - 1) / rb) / nsm);
    const int part = (int)(per_sm % 3);
    const double units = 3.0 * (double)(per_sm / 3) + (part == 1 ? c.one : part == 2 ? c.two : 0.0);
    if (units * (rb + c.start) < cost) {
      cost = units * (rb + c.start);
      best = rb;
    }
  }
  return best;
}

}  // namespace chgpu
