// Forward attention for few query rows per KV head (decode, speculative and short chunked prefill).
//
// With a handful of query tokens the call reads K and V once and does almost nothing with them: it
// is bound by HBM, and the 128-row Q tiles of fwd_ws.cu are the wrong shape for it -- nearly all of
// their rows are padding, and one CTA per SM has a K/V tile or two in flight.  Here the G query heads
// that share a KV head and the Nq tokens form the rows of ONE item (row = token * G + head), so K/V
// cross the SM once for all of them, in blocks of 16 rows, and two CTAs share an SM:
//
//   item      = (batch, KV head, block of 16*RG rows);  T tiles of 64 keys each
//   CTA       = a contiguous range of the tiles of all items, the same length for every CTA of the
//               launch; plan_decode (plan.cu) says how many and which calls come here at all
//   warp 4    TMA producer: K and V boxes (64 keys, 128-byte swizzle) through a ring, 96 KB deep (64 KB at D = 64),
//             192 KB (128 KB) in flight per SM
//   warps 0-3 16 rows x (16*RG keys of the tile) each: RG row groups x 4/RG key groups, each warp
//             with its own running (m, l, O) in registers -- no CTA-wide step inside the loop
//
// The products run as mma.sync m16n8k16 out of ldmatrix: at most 64 rows, about a third of the
// tensor work that would bind before HBM does, and P never leaves its registers, where a tcgen05
// tile would pay the TMEM round trip (S -> registers -> P -> TMEM) of every 64 keys in latency.
//
// A CTA whose range cuts an item leaves (un-normalised O, m, l) of its piece in scratch and counts
// itself in; the CTA that counts in last folds the pieces and writes the rows.  Nobody waits.
//
// Measured (B200, 16 requests, 32/8 heads, 1 token against 4001 keys, D=128 bf16, 262 MB of K/V): 183 us
// through fwd_ws.cu before that packed heads, 48 now, 45.6 us here = 5.7 TB/s, 0.88 of the measured copy bandwidth.  Short
// calls are bound by their ends: with 64-bit divisions for a CTA's range and for every tile, and the first copies
// after the CTA's first synchronisation, 32/8 heads of 500 keys took 8.1 us (6.1 now; D = 64 6.6 and 4.7), 4 x 32/8 heads of
// 1024 9.4 (8.5), 64 items of 9000 at D = 64 27.6 (27.2), all with K and V in L2; calls of 40 us and more are as they were.
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "launch.cuh"
#include "ptx.cuh"

namespace ma {

namespace {

constexpr int kDecThreads = 160;
constexpr int kDecKeys = 64;            // keys per tile
constexpr int kDecBox = kDecKeys * 128; // one [64 keys x 128 B] box
constexpr float kDecLazy = 8.0f;        // log2 units, as in fwd_ws.cu
constexpr int kMergePitch = 36;         // floats per row of the merge buffer (32 + padding)

template <int D>
struct DecLayout {
  static constexpr int kBoxes = D / 64;
  static constexpr int kStageBytes = 2 * kBoxes * kDecBox;  // K then V
  // 64 KB of ring at D = 64 is enough, and more in flight wears on HBM: 64 items of 36002 keys 30.7 us in 96 KB, 29.5 in
  // 64, 16 items of 30000 26.7 / 25.8.  At D = 128 a stage is 32 KB.
  static constexpr int kStages = D == 64 ? 4 : 3;
  static constexpr int kOffMerge = kStages * kStageBytes;   // float[4 warps][16][kMergePitch]
  static constexpr int kOffMl = kOffMerge + 4 * 16 * kMergePitch * 4;  // float2[4 warps][16]
  static constexpr int kOffBar = kOffMl + 4 * 16 * 8;       // full[kStages], empty[kStages]
  static constexpr int kOffMisc = kOffBar + 2 * kStages * 8;  // abort flag, arrival order
  static constexpr int kBytes = kOffMisc + 16;
  static constexpr int kDynSmem = kBytes + 1024;
};

__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
template <bool BF16>
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (BF16)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void workers_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// weight of a partial with maximum m under the total maximum mt (0 for a partial without keys)
__device__ __forceinline__ float part_weight(float m, float mt) {
  return m == -INFINITY ? 0.f : ex2(m - mt);
}

}  // namespace

template <int D, bool BF16, int RG>
__global__ void __launch_bounds__(kDecThreads, 2)
fwd_decode_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                  const DecodeArgs a) {
  using L = DecLayout<D>;
  constexpr int KG = 4 / RG;         // key groups: warps that share a row group
  constexpr int kRows = 16 * RG;     // rows of an item
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;
  uint8_t* gbase = smem_raw + (sbase - raw);
  const uint32_t bars = sbase + L::kOffBar;
  auto full = [&](int s) -> uint32_t { return bars + 8u * s; };
  auto empty = [&](int s) -> uint32_t { return bars + 8u * (L::kStages + s); };
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + L::kOffMisc);
  volatile int* order = abort_flag + 1;

  grid_dep_launch();
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const WaitCtx wc{abort_flag, a.status, MINIATTN_WAIT_LIMIT_NS};
  // this CTA's tiles [lo, hi) of the launch's total
  const long long n_ctas = gridDim.x;
  auto first_tile = [&](long long cta) -> long long {
    return a.small ? div_by(static_cast<int>(cta * a.total), a.by_ctas) : cta * a.total / n_ctas;
  };
  auto item_of = [&](long long x) -> int {
    return a.small ? div_by(static_cast<int>(x), a.by_tiles) : static_cast<int>(x / a.tiles);
  };
  auto cta_of = [&](long long x) -> long long {  // that holds tile x
    return a.small ? div_by(static_cast<int>((x + 1) * n_ctas - 1), a.by_total) : ((x + 1) * n_ctas - 1) / a.total;
  };
  const long long lo = first_tile(blockIdx.x), hi = first_tile(blockIdx.x + 1ll);

  if (warp == 4) {
    // =========================== TMA producer ====================================
    // The whole warp, one elected thread issues (a diverged thread takes several times as long), and it starts as
    // soon as its barriers are there: the first stages are on their way while the workers fetch Q.
    const bool issuer = elect_one();
    if (issuer) {
      for (int s = 0; s < L::kStages; ++s) {
        mbar_init(full(s), 1);
        mbar_init(empty(s), 4);
      }
      *abort_flag = 0;
      fence_mbar_init();
      fence_proxy_async_smem();
      prefetch_tmap(&tm_k);
      prefetch_tmap(&tm_v);
    }
    __syncwarp();
    asm volatile("bar.arrive 2, 160;" ::: "memory");  // the workers look at the barriers from here on
    grid_dep_wait();
    int item = item_of(lo), t = static_cast<int>(lo - static_cast<long long>(item) * a.tiles);
    int b, hk;
    auto locate = [&]() {
      const int kvh = div_by(item, a.by_rb);
      b = div_by(kvh, a.by_hkv);
      hk = kvh - b * a.Hkv;
    };
    locate();
    int slot = 0, par = 1, i = 0;
    for (long long x = lo; x < hi; ++x, ++i) {
      if (i >= L::kStages) mbar_wait(empty(slot), par, wc, kErrWaitFree);
      if (issuer) {
        mbar_expect_tx(full(slot), L::kStageBytes);
        const uint32_t dst = sbase + slot * L::kStageBytes;
#pragma unroll
        for (int bx = 0; bx < L::kBoxes; ++bx)
          tma_load_4d(dst + bx * kDecBox, &tm_k, full(slot), bx * 64, t * kDecKeys, hk, b);
#pragma unroll
        for (int bx = 0; bx < L::kBoxes; ++bx)
          tma_load_4d(dst + (L::kBoxes + bx) * kDecBox, &tm_v, full(slot), bx * 64, t * kDecKeys, hk, b);
      }
      __syncwarp();
      if (++slot == L::kStages) {
        slot = 0;
        par ^= 1;
      }
      if (++t == a.tiles) {
        t = 0;
        ++item;
        locate();
      }
    }
    // give-up path: let the copies in flight land (bounded) before the shared memory is released
    if (*abort_flag) {
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) {
      }
    }
    __syncwarp();
    return;
  }
  grid_dep_wait();
  bool barriers_there = false;

  // ---------------------------------------------------------------- workers
  const int rg = warp % RG, kg = warp / RG;
  const int g = lane >> 2, tig = lane & 3;
  float* merge = reinterpret_cast<float*>(gbase + L::kOffMerge);
  float2* ml_s = reinterpret_cast<float2*>(gbase + L::kOffMl);
  const float c = a.scale_log2;
  // ldmatrix row addresses: lanes 0-7 / 8-15 / 16-23 / 24-31 address the four 8x8 matrices
  const int k_row = (lane & 7) + ((lane >> 4) << 3), k_chunk = (lane >> 3) & 1;        // K: keys x dims
  const int v_row = (lane & 7) + (((lane >> 3) & 1) << 3), v_chunk = lane >> 4;         // V: trans
  int i = 0;  // ring index

  for (long long x = lo; x < hi;) {
    const int item = item_of(x);
    const long long item0 = static_cast<long long>(item) * a.tiles;
    const int t0 = static_cast<int>(x - item0);
    const int t1 = static_cast<int>(min(static_cast<long long>(a.tiles), hi - item0));
    const int kvh = div_by(item, a.by_rb), rb = item - kvh * a.n_rb;
    const int b = div_by(kvh, a.by_hkv), hk = kvh - b * a.Hkv;
    const int row0 = rb * kRows;

    // Q fragments of this warp's 16 rows, and how many keys its two rows of this lane may see.  Ordinary
    // loads, not the read-only kind: the kernel before this one may write Q while this one already runs, and with
    // o = q this one writes it.  (Past L1 they cost 2 us of 24 at 4 tokens of 64/8 heads: four warps share the rows.)
    uint32_t qf[D / 16][4];
    int vis[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int r = row0 + rg * 16 + g + 8 * e;
      const int tok = div_by(r, a.by_g);
      long long v = a.Nk;
      if (a.causal) v = min(v, a.diag + tok + 1);
      const bool ok = r < a.rows;
      vis[e] = ok ? static_cast<int>(max(0ll, v)) : 0;
      const uint16_t* qp = a.q + b * a.qs[0] + (hk * a.G + (r - tok * a.G)) * a.qs[1] + tok * a.qs[2];
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
        const int col = ks * 16 + tig * 2;  // D = 96 runs on the D = 128 kernel: columns past it are 0
        qf[ks][e] = (ok && col < a.D) ? *reinterpret_cast<const uint32_t*>(qp + col) : 0u;
        qf[ks][2 + e] = (ok && col + 8 < a.D) ? *reinterpret_cast<const uint32_t*>(qp + col + 8) : 0u;
      }
    }
    const int vis_min = __reduce_min_sync(0xffffffffu, min(vis[0], vis[1]));

    float acc[D / 8][4];
#pragma unroll
    for (int n = 0; n < D / 8; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[n][e] = 0.f;
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
    if (!barriers_there) asm volatile("bar.sync 2, 160;" ::: "memory");
    barriers_there = true;

    for (int t = t0; t < t1; ++t, ++i) {
      const int slot = i % L::kStages;
      mbar_wait(full(slot), (i / L::kStages) & 1, wc, kErrWaitKV);
      const uint32_t sK = sbase + slot * L::kStageBytes;
      const uint32_t sV = sK + L::kBoxes * kDecBox;
      const int key0 = kg * kRows;  // this warp's keys of the tile: [key0, key0 + 16*RG)
      // All RG*2 accumulator chains advance together, and with one row group each is cut in two: an
      // mma.sync waits for the one before it on its chain, and two chains of eight would leave the
      // warp idle most of the time.
      constexpr int kSplit = RG == 1 ? 2 : 1;
      float sp[kSplit][RG][2][4];
#pragma unroll
      for (int u = 0; u < kSplit; ++u)
#pragma unroll
        for (int kc = 0; kc < RG; ++kc)
#pragma unroll
          for (int e = 0; e < 4; ++e) sp[u][kc][0][e] = sp[u][kc][1][e] = 0.f;
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
#pragma unroll
        for (int kc = 0; kc < RG; ++kc) {
          const int r = key0 + kc * 16 + k_row;
          uint32_t kb[4];
          ldsm4(sK + r * 128 + (ks >> 2) * kDecBox + ((((ks & 3) * 2 + k_chunk) ^ (r & 7)) << 4), kb);
          mma16816<BF16>(sp[ks % kSplit][kc][0], qf[ks], kb[0], kb[1]);
          mma16816<BF16>(sp[ks % kSplit][kc][1], qf[ks], kb[2], kb[3]);
        }
      }
      auto& s = sp[0];
      if constexpr (kSplit == 2) {
#pragma unroll
        for (int kc = 0; kc < RG; ++kc)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            s[kc][0][e] += sp[kSplit - 1][kc][0][e];
            s[kc][1][e] += sp[kSplit - 1][kc][1][e];
          }
      }
      const int kbase = t * kDecKeys + key0;
      if (kbase + kRows > vis_min) {  // diagonal, ragged or padding rows: hide what they must not see
#pragma unroll
        for (int kc = 0; kc < RG; ++kc)
#pragma unroll
          for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (kbase + kc * 16 + n * 8 + tig * 2 + (e & 1) >= vis[e >> 1]) s[kc][n][e] = -INFINITY;
      }
      float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int kc = 0; kc < RG; ++kc)
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          mx[0] = fmax3(mx[0], s[kc][n][0], s[kc][n][1]);
          mx[1] = fmax3(mx[1], s[kc][n][2], s[kc][n][3]);
        }
      bool moved = false;
      float alpha[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], 1));
        mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], 2)) * c;
        const float m_new = fmaxf(m_run[e], mx[e]);
        alpha[e] = 1.f;
        if (m_new - m_run[e] > kDecLazy) {  // also taken when the running maximum is -inf
          alpha[e] = ex2(m_run[e] - m_new);
          m_run[e] = m_new;
          moved = true;
        }
      }
      if (__any_sync(0xffffffffu, moved)) {
        l_run[0] *= alpha[0];
        l_run[1] *= alpha[1];
#pragma unroll
        for (int n = 0; n < D / 8; ++n) {
          acc[n][0] *= alpha[0];
          acc[n][1] *= alpha[0];
          acc[n][2] *= alpha[1];
          acc[n][3] *= alpha[1];
        }
      }
      const float mc0 = m_run[0] == -INFINITY ? 0.f : m_run[0];
      const float mc1 = m_run[1] == -INFINITY ? 0.f : m_run[1];
#pragma unroll
      for (int kc = 0; kc < RG; ++kc) {
        uint32_t pf[4];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const float p0 = ex2(fmaf(s[kc][n][0], c, -mc0)), p1 = ex2(fmaf(s[kc][n][1], c, -mc0));
          const float p2 = ex2(fmaf(s[kc][n][2], c, -mc1)), p3 = ex2(fmaf(s[kc][n][3], c, -mc1));
          l_run[0] += p0 + p1;
          l_run[1] += p2 + p3;
          pf[2 * n] = pack2<BF16>(p0, p1);
          pf[2 * n + 1] = pack2<BF16>(p2, p3);
        }
        const int r = key0 + kc * 16 + v_row;
        const uint32_t rowa = sV + r * 128;
#pragma unroll
        for (int n = 0; n < D / 16; ++n) {
          uint32_t vb[4];
          ldsm4_t(rowa + (n >> 2) * kDecBox + ((((n & 3) * 2 + v_chunk) ^ (r & 7)) << 4), vb);
          mma16816<BF16>(acc[2 * n], pf, vb[0], vb[1]);
          mma16816<BF16>(acc[2 * n + 1], pf, vb[2], vb[3]);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty(slot));
    }

    // ---- end of a piece: fold the key groups, then write the rows or publish the partial ----
    const bool whole = (t0 == 0 && t1 == a.tiles);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      l_run[e] += __shfl_xor_sync(0xffffffffu, l_run[e], 1);
      l_run[e] += __shfl_xor_sync(0xffffffffu, l_run[e], 2);
      if (tig == 0) ml_s[warp * 16 + g + 8 * e] = make_float2(m_run[e], l_run[e]);
    }
    workers_sync();
    float f[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float mt = -INFINITY, lt = 0.f;
#pragma unroll
      for (int k = 0; k < KG; ++k) mt = fmaxf(mt, ml_s[(k * RG + rg) * 16 + g + 8 * e].x);
#pragma unroll
      for (int k = 0; k < KG; ++k) {
        const float2 ml = ml_s[(k * RG + rg) * 16 + g + 8 * e];
        lt += ml.y * part_weight(ml.x, mt);
      }
      f[e] = part_weight(m_run[e], mt);
      if (whole) f[e] *= lt > 0.f ? 1.f / lt : 0.f;
    }
    const long long c_first = whole ? 0 : cta_of(item0);  // CTA that holds the item's tile 0
    const long long my_slot = 2ll * blockIdx.x + (t0 == 0 ? 1 : 0);
    if (tid < kRows && row0 + tid < a.rows) {
      const int rgi = tid >> 4, rr = tid & 15;
      float mt = -INFINITY, lt = 0.f;
      for (int k = 0; k < KG; ++k) mt = fmaxf(mt, ml_s[(k * RG + rgi) * 16 + rr].x);
      for (int k = 0; k < KG; ++k) {
        const float2 ml = ml_s[(k * RG + rgi) * 16 + rr];
        lt += ml.y * part_weight(ml.x, mt);
      }
      if (!whole) {
        a.part_ml[my_slot * kRows + tid] = make_float2(mt, lt);
      } else if (a.lse != nullptr) {
        const int r = row0 + tid, tok = div_by(r, a.by_g), h = hk * a.G + (r - tok * a.G);
        a.lse[(static_cast<long long>(b) * a.Hq + h) * a.Nq + tok] =
            lt > 0.f ? mt * 0.6931471805599453f + __logf(lt) : -INFINITY;
      }
    }
    auto store_row = [&](int r_in, int col, const float4& o) {  // four columns of a finished row
      const int r = row0 + r_in, tok = div_by(r, a.by_g), h = hk * a.G + (r - tok * a.G);
      uint2 w;
      w.x = pack2<BF16>(o.x, o.y);
      w.y = pack2<BF16>(o.z, o.w);
      *reinterpret_cast<uint2*>(a.o + b * a.os[0] + h * a.os[1] + tok * a.os[2] + col) = w;
    };
#pragma unroll
    for (int p = 0; p < D / 32; ++p) {  // 32 columns at a time through 9 KB
      float* mine = merge + warp * 16 * kMergePitch;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int n = p * 4 + j;
        *reinterpret_cast<float2*>(mine + g * kMergePitch + j * 8 + tig * 2) =
            make_float2(acc[n][0] * f[0], acc[n][1] * f[0]);
        *reinterpret_cast<float2*>(mine + (g + 8) * kMergePitch + j * 8 + tig * 2) =
            make_float2(acc[n][2] * f[1], acc[n][3] * f[1]);
      }
      workers_sync();
      const int rr = tid >> 3, c4 = (tid & 7) * 4;
#pragma unroll
      for (int rgi = 0; rgi < RG; ++rgi) {
        const int r_in = rgi * 16 + rr;
        if (row0 + r_in >= a.rows) continue;
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < KG; ++k) {
          const float4 y = *reinterpret_cast<const float4*>(merge + ((k * RG + rgi) * 16 + rr) * kMergePitch + c4);
          o.x += y.x;
          o.y += y.y;
          o.z += y.z;
          o.w += y.w;
        }
        const int col = p * 32 + c4;
        if (!whole) *reinterpret_cast<float4*>(a.part_o + (my_slot * kRows + r_in) * D + col) = o;
        else if (col < a.D) store_row(r_in, col, o);
      }
      workers_sync();
    }
    if (!whole) {
      __threadfence();  // release: the piece before the count
      workers_sync();
      const long long c_last = cta_of(item0 + a.tiles - 1);
      const int n_parts = static_cast<int>(c_last - c_first + 1);
      if (tid == 0) {
        __threadfence();
        *order = atomicAdd(a.counters + c_first, 1);
      }
      workers_sync();
      if (*order == n_parts - 1) {
        __threadfence();  // acquire: every other piece was published before it was counted
        if (tid == 0) a.counters[c_first] = 0;
        const int n_rows = min(kRows, a.rows - row0);
        // total maximum of every row: 128 / kRows threads share a row, each reads every so many-th piece
        constexpr int kPerRow = 128 / kRows;
        {
          const int r_in = tid / kPerRow;
          float m = -INFINITY;
#pragma unroll 4
          for (int p = tid % kPerRow; p < n_parts; p += kPerRow)
            m = fmaxf(m, __ldcg(a.part_ml + (2 * (c_first + p) + (p == 0 ? 1 : 0)) * kRows + r_in).x);
#pragma unroll
          for (int d = kPerRow / 2; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
          if (tid % kPerRow == 0) merge[r_in] = m;  // rows past n_rows read scratch nobody wrote; unused
        }
        workers_sync();
        // `U` groups of four columns a thread at a time, so that their loads are in flight together
        auto fold = [&](auto u_tag) {
          constexpr int U = decltype(u_tag)::value;
          const int n_el = n_rows * (D / 4);
          for (int e0 = tid; e0 < n_el; e0 += 128 * U) {
            float4 o[U];
            float lt[U], mt[U];
            long long at[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const int e = min(e0 + 128 * u, n_el - 1);
              o[u] = make_float4(0.f, 0.f, 0.f, 0.f);
              lt[u] = 0.f;
              mt[u] = merge[e / (D / 4)];
              at[u] = (2 * c_first + 1) * kRows + e / (D / 4);  // the first piece; the others lie at 2*(c_first+p)
            }
#pragma unroll (8 / U)
            for (int p = 0; p < n_parts; ++p) {
#pragma unroll
              for (int u = 0; u < U; ++u) {
                const int col = (min(e0 + 128 * u, n_el - 1) % (D / 4)) * 4;
                const long long i = at[u] + (p == 0 ? 0 : (2 * p - 1) * kRows);
                const float2 ml = __ldcg(a.part_ml + i);
                const float4 y = __ldcg(reinterpret_cast<const float4*>(a.part_o + i * D + col));
                const float w = part_weight(ml.x, mt[u]);
                lt[u] = fmaf(ml.y, w, lt[u]);
                o[u].x = fmaf(y.x, w, o[u].x);
                o[u].y = fmaf(y.y, w, o[u].y);
                o[u].z = fmaf(y.z, w, o[u].z);
                o[u].w = fmaf(y.w, w, o[u].w);
              }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const int e = e0 + 128 * u;
              if (e >= n_el) continue;
              const int r_in = e / (D / 4), col = (e % (D / 4)) * 4;
              const float inv = lt[u] > 0.f ? 1.f / lt[u] : 0.f;
              o[u].x *= inv;
              o[u].y *= inv;
              o[u].z *= inv;
              o[u].w *= inv;
              if (col < a.D) store_row(r_in, col, o[u]);
              if (col == 0 && a.lse != nullptr) {
                const int r = row0 + r_in, tok = div_by(r, a.by_g), h = hk * a.G + (r - tok * a.G);
                a.lse[(static_cast<long long>(b) * a.Hq + h) * a.Nq + tok] =
                    lt[u] > 0.f ? mt[u] * 0.6931471805599453f + __logf(lt[u]) : -INFINITY;
              }
            }
          }
        };
        if (n_rows * (D / 4) > 256) fold(std::integral_constant<int, 4>{});
        else fold(std::integral_constant<int, 1>{});
      }
      workers_sync();  // `order` may be written again only when everyone has read it
    }
    x = item0 + t1;
  }
}

// ---------------------------------------------------------------------------------
template <int D, bool BF16, int RG>
static cudaError_t launch_decode_t(const CUtensorMap* tm, const DecodeArgs& a, int n_ctas, cudaStream_t st) {
  auto kern = fwd_decode_kernel<D, BF16, RG>;
  static std::atomic<unsigned long long> smem_set{0};
  cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(kern), DecLayout<D>::kDynSmem, &smem_set);
  if (e != cudaSuccess) return e;
  return launch_overlapped(kern, n_ctas, kDecThreads, DecLayout<D>::kDynSmem, st, tm[0], tm[1], a);
}

template <int D, bool BF16>
static cudaError_t launch_decode_d(const CUtensorMap* tm, const DecodeArgs& a, int rg, int n_ctas, cudaStream_t st) {
  if (rg == 1) return launch_decode_t<D, BF16, 1>(tm, a, n_ctas, st);
  if (rg == 2) return launch_decode_t<D, BF16, 2>(tm, a, n_ctas, st);
  return launch_decode_t<D, BF16, 4>(tm, a, n_ctas, st);
}

// tm[0], tm[1]: K and V maps with boxes of 64 columns x 64 keys.
cudaError_t launch_fwd_decode(int D, bool bf16, const CUtensorMap* tm, const DecodeArgs& a, int rg, int n_ctas,
                              cudaStream_t st) {
  if (D == 128)
    return bf16 ? launch_decode_d<128, true>(tm, a, rg, n_ctas, st) : launch_decode_d<128, false>(tm, a, rg, n_ctas, st);
  if (D == 64)
    return bf16 ? launch_decode_d<64, true>(tm, a, rg, n_ctas, st) : launch_decode_d<64, false>(tm, a, rg, n_ctas, st);
  return cudaErrorInvalidValue;
}

}  // namespace ma
