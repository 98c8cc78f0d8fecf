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

}  // namespace ma
