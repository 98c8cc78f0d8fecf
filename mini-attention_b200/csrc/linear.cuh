// Arguments of linear.cu, shared with the host launcher.
#pragma once
#include "common.cuh"

namespace ma {

constexpr int kLinearMax = 3;      // weights of one launch
constexpr int kLinearMaxBn = 256;  // columns of a tile (two accumulators fill TMEM)
constexpr int kLinearMaxN = 0x7fffffff - kLinearMaxBn;  // a tile's last column fits 32 bits
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
//
// pays: against a library GEMM for each weight, which reaches 0.92 of the tensor rate and, like this launch, takes about
// 3700 clk beside its work.  q = this estimate / that.  Measured on 98 shapes of GQA_Flash and MHA (bf16, 128 to 16384
// tokens, 64 to 4096 wide), chains of six modules replayed as a graph in bursts / for 0.1 s at the power cap, x's projections in
// one launch over the layers' own calls, the whole module's time:
//   q up to 1             0.84 to 1.02 / 0.82 to 1.02, mean 0.93: taken
//   q up to 1.06          0.90 to 1.02 / 0.90 to 1.08, mean 0.98: taken, but with more than 32 MB of weights
//                         1.01 to 1.03 / 1.06 to 1.11 (4096 wide: every pair fetches its operands itself through L2): not taken
//   q above               0.94 to 1.17 / 0.94 to 1.32, mean 1.01: not taken, but for launches of up to 24000 clk (13 us), 0.94 to
//                         1.02: a module of such launches is bound by the host
// One weight alone saves no launch, and the library's tiles are the better ones: the output projection in this form
// 0.97 to 1.12 of the module, mean 1.03.  It is quicker to issue, though, and a module of up to about 60 us on the GPU is bound by
// that: 2 x 1024 tokens, 16/4 heads of 128 65 us with the layers' calls, 61 with x's projections in one launch, 54 with the
// output's as well, 52 to 57 on the GPU.  So launches of up to 24000 clk, which are those of such modules, are taken.  (Only
// after x's: one of this form between library calls takes the host 3 us more.)
// The answer is the same in a stream that is being captured, although a replay pays no host time: a library that the calls before
// the capture never reached cannot be set up in one.
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
  double weights = 0.;
  for (int i = 0; i < n_seg; ++i) weights += static_cast<double>(N[i]) * K;
  const double launch = 3700.;
  const double own = best + launch, library = M * weights / (2. * pairs * 4096. * 0.92) + n_seg * launch;
  const bool quicker = n_seg > 1 && (own <= library || (own <= 1.06 * library && 2. * weights <= 32e6));
  *pays = K <= 1 << 24 && (quicker || own <= 24000.);
  return bn;
}

}  // namespace ma
