// Projections of the attention modules: y_i = x w_i^T + b_i for up to kLinearMax weights that share x, in one launch.
//
// Two CTAs on neighbouring SMs (a cluster of two) compute a tile of 256 rows x `bn` columns with tcgen05.mma over the pair
// (cta_group::2, M = 256): each holds 128 rows of x and half of the weight's rows, 64 columns of K a stage.  A pair
// walks its tiles with the accumulators in two halves of TMEM, so that a tile is stored while the next is computed.
//
//   warps 0-7   epilogue: accumulator row + bias -> 16 bit -> shared memory -> TMA store, 16 columns at a time
//   warp 8      MMA issuer (in the CTA of rank 0)
//   warp 9      TMA producer (one in each CTA)
//
// The tile's width is the host's choice (a multiple of 16): what leaves the fewest clocks in the last round of tiles.
// 2048 rows, K = 2048 into 2048 + 1024 columns: 18 x 8 tiles of 176 columns are 1.95 rounds of 74 pairs, 12 x 8 of 256
// would be two rounds for 1.3.
#include <atomic>

#include "common.cuh"
#include "launch.cuh"
#include "linear.cuh"
#include "ptx.cuh"

namespace ma {

namespace {

constexpr int kThreads = 320;
constexpr int kWarpMma = 8, kWarpTma = 9;
constexpr int kRows = 128;            // rows of x in one CTA
constexpr int kK = 64;                // columns of K in a stage
constexpr int kStages = 6;
constexpr int kABytes = kRows * kK * 2;
constexpr int kBBytes = kLinearMaxBn / 2 * kK * 2;
constexpr int kStageBytes = kABytes + kBBytes;
constexpr int kStoreCols = 16;        // columns of a store box: 32 rows x 32 bytes
constexpr int kStoreBytes = 32 * kStoreCols * 2;
constexpr int kOffStore = kStages * kStageBytes;
constexpr int kOffBar = kOffStore + 8 * kStoreBufs * kStoreBytes;
constexpr int kBarFull = 0, kBarEmpty = kStages, kBarAccFull = 2 * kStages, kBarAccFree = kBarAccFull + 2;
constexpr int kNumBars = kBarAccFree + 2;
constexpr int kOffMisc = kOffBar + kNumBars * 8;
constexpr int kDynSmem = kOffMisc + 32 + 1024;
static_assert(kDynSmem <= 232448, "shared memory of one SM");

template <bool BF16>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
linear_kernel(const __grid_constant__ LinearArgs a) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t pad = (1024u - (raw & 1023u)) & 1023u;  // the same in both CTAs
  const uint32_t sbase = raw + pad;
  uint8_t* gbase = smem_raw + pad;
  const uint32_t bars = sbase + kOffBar;
  auto bar = [&](int i) -> uint32_t { return bars + 8u * i; };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gbase + kOffMisc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + kOffMisc + 8);

  grid_dep_launch();
  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lane = tid & 31;
  const int rank = static_cast<int>(cluster_rank());
  const int first = blockIdx.x >> 1, step = gridDim.x >> 1;
  const int n_k = (a.K - 1) / kK + 1;

  if (warp == kWarpTma) {
    for (int i = lane; i < kNumBars; i += 32) mbar_init(bar(i), i >= kBarAccFree ? 16 : 1);
    if (lane == 0) *abort_flag = 0;
    fence_mbar_init();
    __syncwarp();
  }
  if (warp == kWarpMma) tmem_alloc_pair(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
  tc_fence_before();
  __syncwarp();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  grid_dep_wait();
  const WaitCtx wc{abort_flag, a.status, MINIATTN_WAIT_LIMIT_NS};

  // tile -> rows and columns: row tiles fastest, so that the pairs at work share few rows of the weights
  auto locate = [&](int tile, int* m0, int* seg, int* n0) {
    const int nt = div_by(tile, a.by_m_tiles);
    *m0 = (tile - nt * static_cast<int>(a.by_m_tiles.d)) * 2 * kRows;
    int s = 0;
#pragma unroll
    for (int i = 1; i < kLinearMax; ++i)
      if (i < a.n_seg && nt >= a.first_tile[i]) s = i;
    *seg = s;
    *n0 = (nt - a.first_tile[s]) * a.bn;
  };

  if (warp < 8) {
    // =========================== epilogue ==========================================
    const int quad = warp & 3, half = warp >> 2;  // 32 rows; even or odd boxes of 16 columns
    const uint32_t stage = sbase + kOffStore + warp * kStoreBufs * kStoreBytes;
    const uint32_t acc_free = mapa(bar(kBarAccFree), 0);
    const int n_box = a.bn / kStoreCols;
    int done = 0;  // tiles of this pair so far
    StoreTurn turn;
    for (int tile = first; tile < a.n_tiles; tile += step, ++done) {
      int m0, seg, n0;
      locate(tile, &m0, &seg, &n0);
      const int buf = done & 1;
      const CUtensorMap* tm = &a.seg[seg].tm_y;
      const uint16_t* bias = a.seg[seg].bias;
      const int n = a.seg[seg].N;
      mbar_wait(bar(kBarAccFull + buf), (done >> 1) & 1, wc, kErrWaitS);
      tc_fence_after();
      const uint32_t tA = tmem_base + buf * 256 + (static_cast<uint32_t>(quad * 32) << 16);
      for (int bx = half; bx < n_box; bx += 2) {
        const int col = n0 + bx * kStoreCols;
        if (col >= n) break;
        uint32_t u[16];
        tmem_ld16(tA + bx * kStoreCols, u);
        float bv[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) bv[i] = 0.f;
        if (bias != nullptr) {  // the same 16 for the whole warp
          if (col + 16 <= n && a.seg[seg].bias_16) {
            const uint4 lo = *reinterpret_cast<const uint4*>(bias + col), hi = *reinterpret_cast<const uint4*>(bias + col + 8);
            const uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float2 f = unpack2<BF16>(w[i]);
              bv[2 * i] = f.x;
              bv[2 * i + 1] = f.y;
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (col + i < n) bv[i] = unpack2<BF16>(bias[col + i]).x;
          }
        }
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
          w[i] = pack2<BF16>(__uint_as_float(u[2 * i]) + bv[2 * i], __uint_as_float(u[2 * i + 1]) + bv[2 * i + 1]);
        const uint32_t box = stage + turn.take() * kStoreBytes;
        if (lane == 0) tma_store_wait_read<kStoreBufs - 1>();
        __syncwarp();
        const uint32_t at = box + lane * (kStoreCols * 2);
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + 16), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          const int row = m0 + rank * kRows + quad * 32;
          if (row < a.M) tma_store_2d(tm, box, col, row);
          tma_store_commit();
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(acc_free + 8 * buf);
    }
    if (lane == 0) tma_store_wait_read0();
  } else if (warp == kWarpMma && rank == 0) {
    // =========================== MMA issuer ========================================
    const uint32_t idesc = make_idesc(1, BF16 ? 1 : 0, 0, 0, 2 * kRows, a.bn);
    const bool issuer = elect_one();
    const uint64_t a_desc = make_smem_desc(sbase, 16, 1024), b_desc = make_smem_desc(sbase + kABytes, 16, 1024);
    int stage = 0, par = 0, done = 0;
    for (int tile = first; tile < a.n_tiles; tile += step, ++done) {
      const int buf = done & 1;
      if (done >= 2) mbar_wait(bar(kBarAccFree + buf), ((done >> 1) - 1) & 1, wc, kErrWaitO);
      tc_fence_after();
      const uint32_t d = tmem_base + buf * 256;
      for (int k = 0; k < n_k; ++k) {
        mbar_wait(bar(kBarFull + stage), par, wc, kErrWaitKV);
        tc_fence_after();
        if (issuer) {
          const uint32_t at = stage * (kStageBytes >> 4);
#pragma unroll
          for (int kk = 0; kk < kK / 16; ++kk)
            mma_f16_ss_pair(d, a_desc + at + kk * 2, b_desc + at + kk * 2, idesc, (k > 0 || kk > 0) ? 1u : 0u);
          mma_commit_pair(bar(kBarEmpty + stage));
          if (k == n_k - 1) mma_commit_pair(bar(kBarAccFull + buf));
        }
        __syncwarp();
        if (++stage == kStages) {
          stage = 0;
          par ^= 1;
        }
      }
    }
  } else if (warp == kWarpTma) {
    // =========================== TMA producer ======================================
    const bool issuer = elect_one();
    const uint32_t full = mapa(bar(kBarFull), 0);
    const int b_rows = a.bn / 2;
    int stage = 0, par = 1, laps = 0;
    for (int tile = first; tile < a.n_tiles; tile += step) {
      int m0, seg, n0;
      locate(tile, &m0, &seg, &n0);
      for (int k = 0; k < n_k; ++k) {
        if (laps > 0) mbar_wait(bar(kBarEmpty + stage), par, wc, kErrWaitFree);
        if (issuer) {
          const uint32_t dst = sbase + stage * kStageBytes;
          if (rank == 0) mbar_expect_tx(bar(kBarFull + stage), 2 * (kABytes + b_rows * kK * 2));
          tma_load_2d_pair(dst, &a.tm_x, full + 8 * stage, k * kK, m0 + rank * kRows);
          tma_load_2d_pair(dst + kABytes, &a.seg[seg].tm_w, full + 8 * stage, k * kK, n0 + rank * b_rows);
        }
        __syncwarp();
        if (++stage == kStages) {
          stage = 0;
          par ^= 1;
          laps = 1;
        }
      }
    }
    // On the give-up path copies may still be in flight: let them land (bounded) before the CTA's shared
    // memory is released.
    if (*abort_flag) {
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) {
      }
    }
  }

  tc_fence_before();
  __syncwarp();
  cluster_sync();  // neither CTA leaves while the other still reads its shared memory or signals its barriers
  if (warp == kWarpMma) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

}  // namespace

cudaError_t launch_linear(bool bf16, const LinearArgs& a, int pairs, cudaStream_t st) {
  static std::atomic<unsigned long long> smem_set[2] = {};
  const void* kern = bf16 ? reinterpret_cast<const void*>(linear_kernel<true>) : reinterpret_cast<const void*>(linear_kernel<false>);
  cudaError_t e = allow_dynamic_smem(kern, kDynSmem, &smem_set[bf16 ? 1 : 0]);
  if (e != cudaSuccess) return e;
  const unsigned grid = 2u * static_cast<unsigned>(a.n_tiles < pairs ? a.n_tiles : pairs);
  return bf16 ? launch_overlapped(linear_kernel<true>, grid, kThreads, kDynSmem, st, a)
              : launch_overlapped(linear_kernel<false>, grid, kThreads, kDynSmem, st, a);
}

}  // namespace ma
