// Arguments of linear.cu, shared with the host launcher.
#pragma once
#include "common.cuh"

namespace ma {

constexpr int kLinearMax = 3;      // weights of one launch
constexpr int kLinearMaxBn = 256;  // columns of a tile (two accumulators fill TMEM)

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
