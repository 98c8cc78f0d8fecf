// Argument block shared by the forward kernels and the host launcher.
#pragma once
#include <cstdint>
#include <cuda.h>
#include <vector_types.h>

namespace ma {

// n / d for 0 <= n < 2^31 without a division: floor((m' * n) / 2^(32 + shift)) with m' = 2^32 + m the multiple of 1 / d
// rounded up (Granlund and Montgomery, "Division by invariant integers using multiplication", 1994).
struct FastDiv {
  uint32_t d, m, shift;
};
inline FastDiv fast_div(uint32_t d) {
  FastDiv f{d, 0, 0};
  while ((1ull << f.shift) < d) ++f.shift;
  f.m = static_cast<uint32_t>(((((1ull << f.shift) - d) << 32) / d) + 1);
  return f;
}
__host__ __device__ inline int div_by(int n, const FastDiv& f) {
#ifdef __CUDA_ARCH__
  const uint32_t high = __umulhi(static_cast<uint32_t>(n), f.m);
#else
  const uint32_t high = static_cast<uint32_t>((static_cast<uint64_t>(n) * f.m) >> 32);
#endif
  return static_cast<int>((high + static_cast<uint32_t>(n)) >> f.shift);
}

struct FwdArgs {
  float*   lse;        // [B, Hq, Nq] or null
  int32_t* status;     // device word for wait-timeout bits, or null
  long long q_pos0;    // global position of query token 0
  long long k_pos0;    // global position of key token 0
  int Nq, Nk, Hq, Hkv, B;
  int causal;
  int d96;             // head dim 96 on the D = 128 kernels: selects the NARROW form
  float scale;         // softmax scale
  float scale_log2;    // softmax scale * log2(e)
  int pack;            // query heads that share a Q tile: row r of a tile is token r / pack, head r % pack
                       // of the group.  Hq counts such groups (1: plain heads).  See head_pack, api.cu
  int tpt;             // query tokens per Q tile: 128 / pack, rounded down
  int n_q_tiles;       // ceil(Nq / tpt)
  int n_pair_items;    // warp-specialised kernel: CTAs [0, n_pair_items) take two Q tiles each,
                       // the CTAs after them one Q tile each (the tail of the last wave)
  int bh_group;        // work items are ordered in groups of this many consecutive (batch, head)
                       // indices: all Q-tile pairs of a group (latest first, heads fastest) before the
                       // next group.  B*Hq = one group, the default order.  Divides B*Hq.
  // divisors a CTA finds its work with, in the order it needs them (set by set_divisors)
  FastDiv by_group_items, by_group, by_heads, by_gqa, by_pack;
  const float* sq;     // INT8-QK: [B, Hq,  ceil(Nq/128)] Q scales (softmax scale * log2e folded in)
  const float* sk;     // INT8-QK: [B, Hkv, ceil(Nk/128)] K scales
  // Balanced launches only (null otherwise): where CTAs that cover part of an item's key range
  // leave their partial result, and the per-item arrival counters (zero between launches).
  float*  part_o;      // [slot][2 tiles][D/4][128 rows][4] fp32, un-normalised O of a piece
  float2* part_ml;     // [slot][2 tiles][128 rows]: (row maximum in log2 units, row sum)
  int*    counters;    // [cut item][2 tiles][arrived, published]
  // Ring steps only (carry_mode != 0): the rows' running state between launches.
  float*  carry_o;     // [B*Hq*carry_tiles][D/4][128 rows][4] fp32, un-normalised O
  float2* carry_ml;    // [B*Hq*carry_tiles][128 rows]: (row maximum in log2 units, row sum)
  int     carry_mode;  // bit 0: fold the stored state in; bit 1: store the new state, no output
  int     carry_tile0; // the state holds carry_tiles tiles per (batch, head); this launch's first
  int     carry_tiles; // Q tile is number carry_tile0 of them
};

// One CTA of a balanced launch, read from the launch's table (kernel parameter space).
struct PlanEntry {
  uint32_t item;         // index in the heaviest-first item order
  uint16_t t0, t1;       // the CTA covers K/V tiles [t0, t1) of the item
  uint16_t slot0;        // first partial slot of the item (its pieces hold consecutive slots)
  uint8_t  part, nparts; // nparts == 1: whole item, the CTA writes the output itself
  uint32_t counter;      // arrival-counter index of a cut item
};
constexpr int kPlanCap = 768;
struct PlanTable { PlanEntry e[kPlanCap]; };
struct NoPlanTable { int unused; };

// Result of the host-side planner (plan.cu).
struct FwdPlan {
  bool split;            // false: launch the items as they are
  int n_whole;           // CTAs [0, n_whole) take items [0, n_whole) whole
  int n_table;           // the CTAs after them read table.e[cta - n_whole]
  int n_slots;           // partial slots the launch writes
  int n_cut_items;       // items covered by more than one CTA
  float est_plain;       // predicted makespans, in K/V-tile steps of one CTA
  float est_balanced;
  PlanTable table;
};

// Few query rows per KV head (fwd_decode.cu): an item is (batch, KV head, block of rows), its rows are
// token * G + (head of the group); the tiles of all items, one after the other, are cut evenly over the CTAs.
struct DecodeArgs {
  const uint16_t* q;
  uint16_t* o;
  long long qs[3], os[3];  // element strides: batch, head, token
  float*   lse;
  int32_t* status;
  long long diag;          // q_pos0 - k_pos0
  long long total;         // tiles of all items
  int Nq, Nk, Hq, Hkv, G, D, causal;
  int rows;                // G * Nq
  int n_rb;                // row blocks per (batch, KV head)
  int tiles;               // 64-key tiles of an item
  int small;               // total * (CTAs + 1) < 2^31: tiles are found by the divisors below, in 32 bits
  FastDiv by_ctas, by_tiles, by_total, by_rb, by_hkv, by_g;
  float scale_log2;
  float*  part_o;          // [2 * CTAs][rows of an item][D] fp32: pieces of cut items, un-normalised
  float2* part_ml;         // [2 * CTAs][rows of an item]: (row maximum in log2 units, row sum)
  int*    counters;        // [CTAs]: pieces published of the item that starts in that CTA; zero between launches
};
struct DecodePlan {
  int rg;                  // 16-row groups of an item (1, 2 or 4); 0: the call is not one for this kernel
  int n_rb, tiles, n_ctas;
  long long total;
};

constexpr int kTileM = 128;   // query rows per MMA tile (TMEM lanes)
constexpr int kTileN = 128;   // keys per K/V tile
constexpr int kWarpRows = 32;  // rows of a Q tile that one warp stores
constexpr int kBoxCols = 64;  // 16-bit elements per 128-byte swizzled row
constexpr int kBoxBytes = kTileN * 128;  // one [128 rows x 128 B] TMA box

// Work item -> (Q-tile pair, (batch, head) index).  Items walk the (batch, head) indices in groups
// of a.bh_group: within a group the latest Q-tile pair first (the heaviest under a causal mask) and
// heads fastest, so that the CTAs in flight share the K/V of few heads.  Shared by the kernels and
// the host planner.
__host__ __device__ inline void item_to_pair_bh(const FwdArgs& a, int n_pairs, int item, int* pair, int* bh) {
  const int group = div_by(item, a.by_group_items);
  const int within = item - group * static_cast<int>(a.by_group_items.d);
  const int back = div_by(within, a.by_group);
  *pair = n_pairs - 1 - back;
  *bh = group * a.bh_group + within - back * a.bh_group;
}
// After Hq, Hkv, n_q_tiles, bh_group and pack are known.
inline void set_divisors(FwdArgs* a) {
  const long long group_items = static_cast<long long>((a->n_q_tiles + 1) / 2) * a->bh_group;
  a->by_group_items = fast_div(group_items > 0 && group_items < 0x7fffffffll ? static_cast<uint32_t>(group_items) : 1u);
  a->by_group = fast_div(a->bh_group > 0 ? a->bh_group : 1);
  a->by_heads = fast_div(a->Hq > 0 ? a->Hq : 1);
  a->by_gqa = fast_div(a->Hkv > 0 && a->Hq >= a->Hkv ? a->Hq / a->Hkv : 1);
  a->by_pack = fast_div(a->pack > 0 ? a->pack : 1);
}

// Number of K/V tiles the Q tiles whose first token is q0 have to visit (all of them without a mask,
// up to the diagonal of the last row with one).  Shared by the kernels and the host planner.
__host__ __device__ inline int kv_tiles_of(const FwdArgs& a, int q0, int nt) {
  long long kv_end = a.Nk;
  if (a.causal) {
    long long last_row = q0 + nt * a.tpt - 1;
    if (last_row > a.Nq - 1) last_row = a.Nq - 1;
    long long vis = a.q_pos0 + last_row - a.k_pos0 + 1;
    if (vis < kv_end) kv_end = vis;
    if (kv_end < 0) kv_end = 0;
  }
  return static_cast<int>((kv_end + kTileN - 1) / kTileN);
}

}  // namespace ma
