// Arguments of linear.cu, shared with the host launcher.
#pragma once
#include "common.cuh"

namespace ma {

constexpr int kLinearMax = 3;      // weights of one launch
constexpr int kLinearMaxBn = 256;  // columns of a tile (two accumulators fill TMEM)
constexpr int kStoreBufs = 4;      // boxes of an epilogue warp in flight

// The buffer an epilogue warp stages its next box in.  Strictly in turn over all tiles of the warp: before it writes
// one, the warp waits for all its copies but the last kStoreBufs - 1 to have read theirs, and only the copy before those
// had this buffer.  (A turn that began anew with each tile would meet a copy that is still under way wherever a tile
// leaves a warp a number of boxes that kStoreBufs does not divide.)
struct StoreTurn {
  int next = 0;
  __host__ __device__ int take() {
    const int at = next;
    next = at + 1 < kStoreBufs ? at + 1 : 0;
    return at;
  }
};

struct LinearSeg {
  CUtensorMap tm_w;      // [N, K], box = bn / 2 rows x 64 columns, 128-byte swizzle
  CUtensorMap tm_y;      // [M, N], box = 32 rows x 16 columns
  const uint16_t* bias;  // [N] or null
  int N;
  int bias_16;           // 1: it starts on a 16-byte boundary
};
struct LinearArgs {
  CUtensorMap tm_x;      // [M, K], box = 128 rows x 64 columns, 128-byte swizzle
  LinearSeg seg[kLinearMax];
  int32_t* status;
  int M, K, n_seg, bn, n_tiles;
  int first_tile[kLinearMax];  // column tile a weight's columns begin with
  FastDiv by_m_tiles;
};

// Width of a tile: fewest clocks over the rounds of tiles, at bn / 2 clk for 16 columns of K and about 1500 a tile.
// pays: whether that is expected to be no slower than a library GEMM for each weight, which reaches 0.92 of the tensor
// rate at these sizes; either takes about 2 us a launch beside its work.  Measured, us of device time for the whole of
// GQA_Flash in bf16, the layers' own calls / x's projections in one launch / the output's too: 2 x 1024 tokens, 16/4
// heads of 128 52.6 / 49.9 / 50.4 (host-bound without a graph: 90.8 / 81.8 / 56.3); 1 x 4096, 32/8 heads 398 / 377 / 374;
// 4 x 4096, 32/8 1766 / 1581 / 1570; 2 x 777, 24/8, where 1554 rows leave a seventh of the last row tiles 76.0 / 78.6 /
// 83.2: not taken.  A launch of up to 13 us is taken in any case: the calls of the layers then take the host longer
// than the GPU (1 x 512 tokens, 8/2 heads of 64: 66.5 us a call with them, 56.4 without, 16 on the device either way).
// Never with so many columns of K that a tile would come near the bounded waits' limit (about 8 clk a column, 1 s).
inline int linear_tile(int M, int K, int n_seg, const int* N, int pairs, bool* pays) {
  const long long m_tiles = (M + 255ll) / 256;
  long long best = -1;
  int bn = kLinearMaxBn;
  for (int w = kLinearMaxBn; w >= 64; w -= 16) {
    long long tiles = 0;
    for (int i = 0; i < n_seg; ++i) tiles += (N[i] + (w - 1ll)) / w;
    tiles *= m_tiles;
    const long long rounds = (tiles + pairs - 1) / pairs;
    const long long per_mma = w / 2 > 48 ? w / 2 : 48;  // narrower ones wait for shared memory
    const long long clk = rounds * (per_mma * ((K + 15ll) / 16) + 1500);
    if (best < 0 || clk < best) {
      best = clk;
      bn = w;
    }
  }
  double macs = 0.;
  for (int i = 0; i < n_seg; ++i) macs += static_cast<double>(M) * N[i] * K;
  const double launch = 3700.;
  *pays = K <= 1 << 24 &&
          (best + launch <= 1.08 * (macs / (2. * pairs * 4096. * 0.92) + n_seg * launch) ||
           best + launch <= 24000.);
  return bn;
}

}  // namespace ma
