// INT8 pre-pass for the INT8-QK attention variant (no counterpart in the reference code; the
// recipe is the SageAttention-style one of the task configuration):
//   1. K is smoothed: the per-(batch, KV head, channel) mean over tokens is subtracted.  Every
//      score of a row moves by the same amount q.mean(K), so softmax is unchanged.
//   2. Q and the smoothed K are quantised to int8 with one symmetric fp32 scale per block of 128
//      tokens: scale = max|x| / 127 over the 128 x D slab (1 for an all-zero slab),
//      x8 = round-half-even(x / scale), clamped to [-127, 127].
// Two launches: stage 1 quantises Q and sums the columns of K (independent work, one grid), stage 2
// smooths and quantises K.  Stage 2 is launched as a programmatic dependent of stage 1: its CTAs
// become resident while stage 1 drains and load their K slabs before they wait for stage 1's
// column sums, so the second launch's ramp and first loads hide under the first one's tail; stage 1 stands in
// the same relation to the kernel before it, and the attention kernel to stage 2.
// What bounds them: HBM and the loads of a CTA that waits for its own slab, after the instructions were the bound.  With
// one score at a time, a branch for each, a margin around a tie that sent 6 % of the warps' elements through a division, and (bf16)
// the unpacked slab held in registers, the pre-pass took, us fp16 / bf16: 2 x 16 heads, 8192 tokens, D = 64 37.0 / 39.4, now
// 30.7 / 32.6 (134 MB, 4.4 TB/s); 2 x 64/16 heads, 8265, D = 128 144.9 / 214.6, now 117.9 / 132.5 (576 MB, 4.9).
// 16-byte loads, 8-byte int8 stores, one CTA per
// (128-token block, head, batch) or per 1024-token column-sum chunk.  Algorithmic traffic per element: K 2 B (mean pass) + 2 B + 1 B,
// Q 2 B + 1 B, plus 4 B per 128 x D slab for the scale.
// What these kernels read is not declared __restrict__: the compiler would take it for read-only over the whole
// kernel, and the kernel before may still write it while this one already runs (before its grid dependency wait).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

#include "launch.cuh"

namespace ma {

// Scratch of the allocation-free pre-pass entry point (miniattn_quant_qk_int8_static): the
// column sums of K, B * Hkv * ceil(Nk/1024) * D floats, at most kStaticColsumFloats (256 KB).
// Every GPU that loads the library holds this array until the process exits.  In host code the
// name below is only a handle for cudaGetSymbolAddress, never a device address.
constexpr long long kStaticColsumFloats = 65536;
static __device__ __align__(256) float g_static_colsum[kStaticColsumFloats];

namespace {

template <bool BF16>
__device__ __forceinline__ void unpack8(const uint4& w, float (&f)[8]) {
  const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 a;
    if constexpr (BF16) {
      a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u[i]));
    } else {
      a = __half22float2(*reinterpret_cast<const __half2*>(&u[i]));
    }
    f[2 * i] = a.x;
    f[2 * i + 1] = a.y;
  }
}

// Pairs of fp32 in 64-bit registers, low word first: one issue slot for two.  Subnormal numbers are kept, as in the
// scalar operations of the same rounding.
__device__ __forceinline__ uint64_t pair_of(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 halves_of(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t pair_add(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t pair_mul(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t pair_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

constexpr int kSumRows = 1024;  // tokens per partial column sum
constexpr float kNearTie = 1e-4f;
// CTAs of an SM that the registers are made to allow.  Free choice takes 58 (D = 64) and 78 registers, 4 and 3 CTAs; one
// more (48 and 64, a few spilled around the rare division) measured, us for both launches of the pre-pass, fp16 / bf16:
// 2 x 16 heads, 8192 tokens, D = 64 32.2 / 34.5 -> 30.7 / 32.6; 2 x 64/16 heads, 8265, D = 128 122.4 / 138.5 -> 117.9 / 132.5.
// Two more at D = 64 (40 registers) 33.3 / 35.4.
template <int D>
constexpr int kCtasPerSm = D == 64 ? 5 : 4;

}  // namespace

// partial[b, h, chunk, d] = sum over the chunk's tokens of k[b, h, token, d]
template <int D, bool BF16>
__device__ __forceinline__ void colsum_body(const uint16_t* k, long long sb, long long sh,
                                            long long sn, int N, float* __restrict__ partial,
                                            int n_chunks, int chunk, int h, int b, int H) {
  constexpr int CPR = D / 8;          // 16-byte chunks per row
  constexpr int RPP = 256 / CPR;      // rows per pass
  const int col8 = threadIdx.x % CPR, r0 = threadIdx.x / CPR;
  const uint16_t* base = k + b * sb + h * sh;
  uint64_t acc2[4] = {0, 0, 0, 0};
  const int row_end = min(N, (chunk + 1) * kSumRows);
  for (int row = chunk * kSumRows + r0; row < row_end; row += RPP) {
    const uint4 w = *reinterpret_cast<const uint4*>(base + row * sn + col8 * 8);
    float f[8];
    unpack8<BF16>(w, f);
#pragma unroll
    for (int i = 0; i < 4; ++i) acc2[i] = pair_add(acc2[i], pair_of(f[2 * i], f[2 * i + 1]));
  }
  __shared__ __align__(16) float red[RPP][D];
#pragma unroll
  for (int i = 0; i < 4; ++i) *reinterpret_cast<float2*>(&red[r0][col8 * 8 + 2 * i]) = halves_of(acc2[i]);
  __syncthreads();
  if (threadIdx.x < D) {
    float s = 0.f;
#pragma unroll 4
    for (int r = 0; r < RPP; ++r) s += red[r][threadIdx.x];
    partial[((static_cast<long long>(b) * H + h) * n_chunks + chunk) * D + threadIdx.x] = s;
  }
}

// One CTA per (128-token block, head, batch): x8 = round(x' / scale), x' = x - mean (K) or x (Q).
template <int D, bool BF16, bool SMOOTH>
__device__ __forceinline__ void quant_body(const uint16_t* x, long long sb, long long sh,
                                           long long sn, int N, const float* partial,
                                           int n_chunks, int8_t* __restrict__ x8,
                                           float* __restrict__ scale_out, float fold,
                                           float* __restrict__ mean_out, int blk, int h, int b, int H,
                                           int n_blocks) {
  constexpr int CPR = D / 8;
  constexpr int PER = 16 * D / 256;  // chunks per thread (128 rows * D/8 chunks / 256 threads)
  __shared__ __align__(16) float minus_mean[D];
  __shared__ float wmax[8];
  const uint16_t* base = x + b * sb + h * sh;
  // The slab stays in registers as loaded (16-bit pairs) and is unpacked twice, once for the
  // maximum and once for the quantisation: a quarter of the registers of an fp32 copy, so more
  // CTAs (and bytes in flight) fit an SM.  The loads are issued before the channel means are
  // summed, so that the two global-memory latencies overlap.
  uint4 raw[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int id = threadIdx.x + i * 256;
    const int row = blk * 128 + id / CPR, col8 = id % CPR;
    raw[i] = make_uint4(0u, 0u, 0u, 0u);
    if (row < N) raw[i] = *reinterpret_cast<const uint4*>(base + row * sn + col8 * 8);
  }
  if (SMOOTH) {
    // everything above is independent of stage 1; its column sums are complete and visible from here
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();  // the attention kernel's set-up may overlap the rest
    if (threadIdx.x < D) {
      float s = 0.f;
      const float* p = partial + (static_cast<long long>(b) * H + h) * n_chunks * D + threadIdx.x;
      for (int c = 0; c < n_chunks; ++c) s += p[c * D];
      const float m = s / static_cast<float>(N);
      minus_mean[threadIdx.x] = -m;
      if (blk == 0 && mean_out != nullptr) mean_out[(static_cast<long long>(b) * H + h) * D + threadIdx.x] = m;
    }
    __syncthreads();
  }
  auto load = [&](int i, int col8, uint64_t (&x2)[4]) {  // chunk i of this thread, smoothed
    float f[8];
    unpack8<BF16>(raw[i], f);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      x2[e] = pair_of(f[2 * e], f[2 * e + 1]);
      if (SMOOTH) {
        const float2 m = *reinterpret_cast<const float2*>(minus_mean + col8 * 8 + 2 * e);
        x2[e] = pair_add(x2[e], pair_of(m.x, m.y));
      }
    }
  };
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int id = threadIdx.x + i * 256;
    const int row = blk * 128 + id / CPR, col8 = id % CPR;
    if (row < N) {
      uint64_t x2[4];
      load(i, col8, x2);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = halves_of(x2[e]);
        amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = wmax[0];
#pragma unroll
  for (int w = 1; w < 8; ++w) amax = fmaxf(amax, wmax[w]);
  const float scale = amax > 0.f ? __fdiv_rn(amax, 127.f) : 1.f;
  const float inv = __frcp_rn(scale);
  if (threadIdx.x == 0)
    scale_out[(static_cast<long long>(b) * H + h) * n_blocks + blk] = scale * fold;
  int8_t* obase = x8 + ((static_cast<long long>(b) * H + h) * N) * D;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int id = threadIdx.x + i * 256;
    const int row = blk * 128 + id / CPR, col8 = id % CPR;
    if (row < N) {
      // round-half-even(x / scale), bit for bit, without a division per element: y = x * (1/scale) and the rounded
      // quotient are each within 1.6e-5 of the true one, and adding 1.5*2^23 rounds y to the nearest integer (ties to
      // even), whose low byte is then the sum's.  Only where y lies within kNearTie of a tie can the two differ: one
      // element in 5000, one look at the largest distance for eight.
      uint64_t x2[4], sum[4];
      // or the compiler keeps the first pass's fp32 values: 106 instead of 78 registers at D = 128 bf16
      asm volatile("" : "+r"(raw[i].x), "+r"(raw[i].y), "+r"(raw[i].z), "+r"(raw[i].w));
      load(i, col8, x2);
      const uint64_t inv2 = pair_of(inv, inv), big = pair_of(12582912.f, 12582912.f);
      const uint64_t minus_big = pair_of(-12582912.f, -12582912.f), minus_one = pair_of(-1.f, -1.f);
      uint64_t d2[4];
      float far = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint64_t y = pair_mul(x2[e], inv2);
        sum[e] = pair_add(y, big);
        d2[e] = pair_fma(pair_add(sum[e], minus_big), minus_one, y);
        const float2 d = halves_of(d2[e]);
        far = fmaxf(far, fmaxf(fabsf(d.x), fabsf(d.y)));
      }
      uint32_t t[8];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 w = halves_of(sum[e]);
        t[2 * e] = __float_as_uint(w.x);
        t[2 * e + 1] = __float_as_uint(w.y);
      }
      if (far > 0.5f - kNearTie) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float2 d = halves_of(d2[e >> 1]), f = halves_of(x2[e >> 1]);
          if (fabsf((e & 1) ? d.y : d.x) > 0.5f - kNearTie)
            t[e] = static_cast<uint32_t>(max(-127, min(127, __float2int_rn(__fdiv_rn((e & 1) ? f.y : f.x, scale)))));
        }
      }
      const uint32_t lo = __byte_perm(__byte_perm(t[0], t[1], 0x0040), __byte_perm(t[2], t[3], 0x0040), 0x5410);
      const uint32_t hi = __byte_perm(__byte_perm(t[4], t[5], 0x0040), __byte_perm(t[6], t[7], 0x0040), 0x5410);
      *reinterpret_cast<uint2*>(obase + static_cast<long long>(row) * D + col8 * 8) = make_uint2(lo, hi);
    }
  }
}

// Stage 1, one launch: the Q quantiser (nothing depends on it but the attention kernel) and the
// partial column sums of K.  The first gridDim.x - q_blocks blocks sum K, the rest quantise Q.
template <int D, bool BF16>
__global__ void __launch_bounds__(256, kCtasPerSm<D>)
prepass_stage1_kernel(const uint16_t* q, long long qsb, long long qsh, long long qsn, int Nq,
                      int Hq, int nqb, int8_t* __restrict__ q8, float* __restrict__ sq, float fold,
                      const uint16_t* k, long long ksb, long long ksh, long long ksn, int Nk,
                      int Hkv, int nch, float* __restrict__ partial, int q_blocks) {
  // This launch may start while the kernel before it drains (an earlier call's attention still reads the
  // buffers written here).  The dependent launch (stage 2) may start as soon as every CTA of this grid is
  // past that wait, no earlier: it reads K before its own wait.
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  // the column-sum CTAs read eight times as much as a quantiser CTA: they go first
  const int s_blocks = static_cast<int>(gridDim.x) - q_blocks;
  if (static_cast<int>(blockIdx.x) >= s_blocks) {
    const int id = blockIdx.x - s_blocks;
    const int blk = id % nqb, h = (id / nqb) % Hq, b = id / (nqb * Hq);
    quant_body<D, BF16, false>(q, qsb, qsh, qsn, Nq, nullptr, 0, q8, sq, fold, nullptr, blk, h, b, Hq, nqb);
  } else {
    const int c = blockIdx.x;
    const int chunk = c % nch, h = (c / nch) % Hkv, b = c / (nch * Hkv);
    colsum_body<D, BF16>(k, ksb, ksh, ksn, Nk, partial, nch, chunk, h, b, Hkv);
  }
}

// Stage 2: smooth and quantise K (needs every column sum of stage 1).
template <int D, bool BF16>
__global__ void __launch_bounds__(256, kCtasPerSm<D>)
quant_k_kernel(const uint16_t* k, long long sb, long long sh, long long sn, int N,
               const float* partial, int n_chunks, int8_t* __restrict__ k8,
               float* __restrict__ scale_out, float* __restrict__ mean_out) {
  quant_body<D, BF16, true>(k, sb, sh, sn, N, partial, n_chunks, k8, scale_out, 1.0f, mean_out,
                            blockIdx.x, blockIdx.y, blockIdx.z, gridDim.y, gridDim.x);
}

// q8/k8: contiguous [B, H, N, D] int8; scales: [B, H, ceil(N/128)] fp32; partial: scratch of
// B * Hkv * ceil(N/1024) * D floats; k_mean (optional): [B, Hkv, D].
template <int D, bool BF16>
static cudaError_t launch_quant_t(const void* q, const long long* qs, const void* k, const long long* ks,
                                  int B, int Hq, int Hkv, int Nq, int Nk, float q_fold, int8_t* q8,
                                  int8_t* k8, float* sq, float* sk, float* partial, float* k_mean,
                                  cudaStream_t st) {
  const int nqb = (Nq + 127) / 128, nkb = (Nk + 127) / 128, nch = (Nk + kSumRows - 1) / kSumRows;
  const long long q_blocks = static_cast<long long>(nqb) * Hq * B;
  const long long s_blocks = static_cast<long long>(nch) * Hkv * B;
  if (q_blocks + s_blocks > 0x7fffffffll) return cudaErrorInvalidValue;
  if (q_blocks + s_blocks > 0) {
    cudaError_t e = launch_overlapped(prepass_stage1_kernel<D, BF16>, static_cast<unsigned>(q_blocks + s_blocks), 256, 0, st,
                                      static_cast<const uint16_t*>(q), qs[0], qs[1], qs[2], Nq, Hq, nqb, q8, sq, q_fold,
                                      static_cast<const uint16_t*>(k), ks[0], ks[1], ks[2], Nk, Hkv, nch, partial,
                                      static_cast<int>(q_blocks));
    if (e != cudaSuccess) return e;
  }
  if (Nk > 0)
    return launch_overlapped(quant_k_kernel<D, BF16>, dim3(nkb, Hkv, B), 256, 0, st, static_cast<const uint16_t*>(k), ks[0],
                             ks[1], ks[2], Nk, static_cast<const float*>(partial), nch, k8, sk, k_mean);
  return cudaGetLastError();
}

cudaError_t launch_quant_qk(int D, bool bf16, const void* q, const long long* qs, const void* k,
                            const long long* ks, int B, int Hq, int Hkv, int Nq, int Nk, float q_fold,
                            int8_t* q8, int8_t* k8, float* sq, float* sk, float* partial, float* k_mean,
                            cudaStream_t st) {
  if (D == 64)
    return bf16 ? launch_quant_t<64, true>(q, qs, k, ks, B, Hq, Hkv, Nq, Nk, q_fold, q8, k8, sq, sk, partial, k_mean, st)
                : launch_quant_t<64, false>(q, qs, k, ks, B, Hq, Hkv, Nq, Nk, q_fold, q8, k8, sq, sk, partial, k_mean, st);
  if (D == 128)
    return bf16 ? launch_quant_t<128, true>(q, qs, k, ks, B, Hq, Hkv, Nq, Nk, q_fold, q8, k8, sq, sk, partial, k_mean, st)
                : launch_quant_t<128, false>(q, qs, k, ks, B, Hq, Hkv, Nq, Nk, q_fold, q8, k8, sq, sk, partial, k_mean, st);
  return cudaErrorInvalidValue;
}

long long static_colsum_capacity() { return kStaticColsumFloats; }

// Device address of g_static_colsum on the current device, looked up once per device with that
// device current (the first call on a device does the lookup).
static cudaError_t static_colsum_ptr(float** out) {
  static std::mutex mu;
  static float* ptrs[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(mu);
  if (ptrs[dev] == nullptr) {
    float* p = nullptr;
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_static_colsum);
    if (e != cudaSuccess) return e;
    ptrs[dev] = p;
  }
  *out = ptrs[dev];
  return cudaSuccess;
}

// Same pre-pass as launch_quant_qk with the column-sum scratch taken from g_static_colsum.
// Nothing in the array has to start at zero: the column-sum kernel overwrites every entry the
// quantiser reads.  The caller has checked that the problem fits kStaticColsumFloats.
cudaError_t launch_quant_qk_static(int D, bool bf16, const void* q, const long long* qs, const void* k,
                                   const long long* ks, int B, int Hq, int Hkv, int Nq, int Nk,
                                   float q_fold, int8_t* q8, int8_t* k8, float* sq, float* sk,
                                   float* k_mean, cudaStream_t st) {
  float* scratch = nullptr;
  cudaError_t e = static_colsum_ptr(&scratch);
  if (e != cudaSuccess) return e;
  return launch_quant_qk(D, bf16, q, qs, k, ks, B, Hq, Hkv, Nq, Nk, q_fold, q8, k8, sq, sk, scratch,
                         k_mean, st);
}

}  // namespace ma
