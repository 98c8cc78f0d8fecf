// Host side of the C ABI declared in include/miniattn.h: argument validation
// (mirrors the checks of the reference launcher, kernels/flash_attn/cuda/sm_120/kernel/
// flash_attention.cu:41-80, relaxed to "head dim contiguous" instead of fully contiguous),
// TMA tensor-map construction from the caller's strides, kernel selection and launch.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>
#include <vector>

#include "../../include/miniattn.h"
#include "common.cuh"
#include "linear.cuh"

namespace ma {
cudaError_t launch_fwd_simple(int D, bool bf16, const CUtensorMap* tm, const FwdArgs& a,
                              cudaStream_t st);
cudaError_t launch_fwd_ws(int D, bool bf16, const CUtensorMap* tm, const FwdArgs& a, int sm_count,
                          cudaStream_t st);
cudaError_t launch_fwd_ws_int8qk(int D, bool bf16, const CUtensorMap* tm, const FwdArgs& a,
                                 int sm_count, cudaStream_t st);
cudaError_t launch_fwd_ws_plan(int D, bool bf16, bool qk8, const CUtensorMap* tm, const FwdArgs& a,
                               const FwdPlan& plan, cudaStream_t st);
cudaError_t launch_fwd_decode(int D, bool bf16, const CUtensorMap* tm, const DecodeArgs& a, int rg, int n_ctas,
                              cudaStream_t st);
void plan_decode(int B, int Hq, int Hkv, int Nq, int Nk, int D, int causal, long long diag, int sms, bool cut,
                 DecodePlan* d);
bool plan_considered(const FwdArgs& a, int sms);
void plan_fwd(const FwdArgs& a, int D, int sms, FwdPlan* plan);
cudaError_t launch_quant_qk(int D, bool bf16, const void* q, const long long* qs, const void* k,
                            const long long* ks, int B, int Hq, int Hkv, int Nq, int Nk, float q_fold,
                            int8_t* q8, int8_t* k8, float* sq, float* sk, float* partial, float* k_mean,
                            cudaStream_t st);
long long static_colsum_capacity();
cudaError_t launch_quant_qk_static(int D, bool bf16, const void* q, const long long* qs, const void* k,
                                   const long long* ks, int B, int Hq, int Hkv, int Nq, int Nk,
                                   float q_fold, int8_t* q8, int8_t* k8, float* sq, float* sk,
                                   float* k_mean, cudaStream_t st);
cudaError_t launch_linear(bool bf16, const LinearArgs& a, int pairs, cudaStream_t st);
cudaError_t launch_wait_selftest(int32_t* status, unsigned long long limit_ns, cudaStream_t st);
cudaError_t launch_merge_partials(float* acc_o, float* acc_lse, const void* part_o,
                                  const float* part_lse, void* out, long long rows, int D, bool bf16,
                                  int init, long long rows_per_slab, long long out_slab_stride,
                                  int sm_count, cudaStream_t st);
}  // namespace ma

namespace {

thread_local char g_err[512] = "";

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// 4-D map over a [B, H, N, D] logical tensor with arbitrary (batch, head, token) strides:
// dims (fastest first) = (d, token, head, batch); box = 64 x `box_rows` x 1 x 1 elements
// (one 128-byte swizzled row per token).
// Recently encoded maps of the calling thread: a loop that calls the operator on the same tensors
// pays the driver's encoder once (four encodes are about a third of the host time of a launch).
struct MapKey {
  const void* base;
  int64_t stride[3];
  int elem_bytes, dt, D, N, H, B, box_cols, box_rows, swizzle;
  bool operator==(const MapKey& o) const {
    return base == o.base && stride[0] == o.stride[0] && stride[1] == o.stride[1] && stride[2] == o.stride[2] &&
           elem_bytes == o.elem_bytes && dt == o.dt && D == o.D && N == o.N && H == o.H && B == o.B &&
           box_cols == o.box_cols && box_rows == o.box_rows && swizzle == o.swizzle;
  }
};
struct MapSlot {
  MapKey key;
  CUtensorMap map;
  bool valid;
};
constexpr int kMapSlots = 16;

int make_map(CUtensorMap* out, const void* base, int elem_bytes, CUtensorMapDataType dt, int D,
             int N, int H, int B, const int64_t stride[3], int box_cols, int box_rows,
             const char* what, CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B) {
  thread_local MapSlot cache[kMapSlots] = {};
  thread_local unsigned next_slot = 0;
  const MapKey key{base, {stride[0], stride[1], stride[2]}, elem_bytes, static_cast<int>(dt), D, N, H, B,
                   box_cols, box_rows, static_cast<int>(swizzle)};
  for (int i = 0; i < kMapSlots; ++i)
    if (cache[i].valid && cache[i].key == key) {
      *out = cache[i].map;
      return MINIATTN_OK;
    }
  EncodeTiledFn enc = encode_fn();
  if (!enc) return fail(MINIATTN_ECUDA, "cuTensorMapEncodeTiled entry point not found");
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)N, (cuuint64_t)H, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)stride[2] * elem_bytes, (cuuint64_t)stride[1] * elem_bytes,
                           (cuuint64_t)stride[0] * elem_bytes};
  cuuint32_t box[4] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  // a size-1 dim may carry any stride; give the encoder a legal one
  for (int i = 0; i < 3; ++i)
    if (dims[i + 1] == 1) strides[i] = (cuuint64_t)D * elem_bytes;
  CUresult r = enc(out, dt, 4, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return fail(MINIATTN_ECUDA, "cuTensorMapEncodeTiled(%s) failed with CUresult %d", what, (int)r);
  MapSlot& slot = cache[next_slot++ % kMapSlots];
  slot.key = key;
  slot.map = *out;
  slot.valid = true;
  return MINIATTN_OK;
}

// Q or O for fwd_ws.cu: dims (fastest first) = (d, head of a group of `pack`, token, group, batch);
// box = 64 x pack x tpt x 1 x 1, so that a tile's rows are (token, head) with the head fastest.
int make_map_packed(CUtensorMap* out, const void* base, CUtensorMapDataType dt, int D, int N, int groups, int B,
                    const int64_t stride[3], int pack, int tpt, const char* what) {
  thread_local MapSlot cache[kMapSlots] = {};
  thread_local unsigned next_slot = 0;
  const MapKey key{base, {stride[0], stride[1], stride[2]}, pack, static_cast<int>(dt), D, N, groups, B, tpt, 0, 0};
  for (int i = 0; i < kMapSlots; ++i)
    if (cache[i].valid && cache[i].key == key) {
      *out = cache[i].map;
      return MINIATTN_OK;
    }
  EncodeTiledFn enc = encode_fn();
  if (!enc) return fail(MINIATTN_ECUDA, "cuTensorMapEncodeTiled entry point not found");
  cuuint64_t dims[5] = {(cuuint64_t)D, (cuuint64_t)pack, (cuuint64_t)N, (cuuint64_t)groups, (cuuint64_t)B};
  cuuint64_t strides[4] = {(cuuint64_t)stride[1] * 2, (cuuint64_t)stride[2] * 2, (cuuint64_t)stride[1] * pack * 2,
                           (cuuint64_t)stride[0] * 2};
  cuuint32_t box[5] = {ma::kBoxCols, (cuuint32_t)pack, (cuuint32_t)tpt, 1, 1};
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  // a size-1 dim may carry any stride; give the encoder a legal one
  for (int i = 0; i < 4; ++i)
    if (dims[i + 1] == 1) strides[i] = (cuuint64_t)D * 2;
  CUresult r = enc(out, dt, 5, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return fail(MINIATTN_ECUDA, "cuTensorMapEncodeTiled(%s) failed with CUresult %d", what, (int)r);
  MapSlot& slot = cache[next_slot++ % kMapSlots];
  slot.key = key;
  slot.map = *out;
  slot.valid = true;
  return MINIATTN_OK;
}

// 2-D map over a row-major [rows, cols] matrix of 16-bit elements, for linear.cu.
int make_map_2d(CUtensorMap* out, const void* base, CUtensorMapDataType dt, int rows, int cols, int64_t ld, int box_rows,
                int box_cols, CUtensorMapSwizzle swizzle, const char* what) {
  thread_local MapSlot cache[kMapSlots] = {};
  thread_local unsigned next_slot = 0;
  const MapKey key{base, {ld, 0, 0}, 2, static_cast<int>(dt), cols, rows, 1, 1, box_cols, box_rows, static_cast<int>(swizzle)};
  for (int i = 0; i < kMapSlots; ++i)
    if (cache[i].valid && cache[i].key == key) {
      *out = cache[i].map;
      return MINIATTN_OK;
    }
  EncodeTiledFn enc = encode_fn();
  if (!enc) return fail(MINIATTN_ECUDA, "cuTensorMapEncodeTiled entry point not found");
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)(rows == 1 ? cols : ld) * 2};  // a size-1 dim may carry any stride
  cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(out, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return fail(MINIATTN_ECUDA, "cuTensorMapEncodeTiled(%s) failed with CUresult %d", what, (int)r);
  MapSlot& slot = cache[next_slot++ % kMapSlots];
  slot.key = key;
  slot.map = *out;
  slot.valid = true;
  return MINIATTN_OK;
}

int check_tensor(const void* p, const int64_t s[3], int D, const char* name) {
  if (p == nullptr) return fail(MINIATTN_EINVAL, "%s is null", name);
  if (reinterpret_cast<uintptr_t>(p) % 16 != 0)
    return fail(MINIATTN_EINVAL, "%s must be 16-byte aligned", name);
  for (int i = 0; i < 3; ++i) {
    if (s[i] < 0) return fail(MINIATTN_EINVAL, "%s has a negative stride", name);
    if (s[i] % 8 != 0)
      return fail(MINIATTN_EINVAL, "%s stride %d (%lld) is not a multiple of 8 elements", name, i,
                  (long long)s[i]);
  }
  if (s[2] < D) return fail(MINIATTN_EINVAL, "%s token stride is smaller than D", name);
  return MINIATTN_OK;
}

int device_sm_count(int* sms, int* major) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail(MINIATTN_ECUDA, "cudaGetDevice: %s", cudaGetErrorString(e));
  // one entry per device ordinal, filled on first use under a lock (host threads may drive
  // different devices at the same time)
  constexpr int kMaxDevices = 64;
  static std::mutex mu;
  static int table_sms[kMaxDevices] = {0};
  static int table_major[kMaxDevices] = {0};
  if (dev < 0 || dev >= kMaxDevices) return fail(MINIATTN_EUNSUPPORTED, "device ordinal %d out of range", dev);
  std::lock_guard<std::mutex> g(mu);
  if (table_sms[dev] == 0) {
    int n = 0, mj = 0;
    if ((e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&mj, cudaDevAttrComputeCapabilityMajor, dev)) != cudaSuccess)
      return fail(MINIATTN_ECUDA, "cudaDeviceGetAttribute: %s", cudaGetErrorString(e));
    table_sms[dev] = n;
    table_major[dev] = mj;
  }
  *sms = table_sms[dev];
  *major = table_major[dev];
  return MINIATTN_OK;
}

}  // namespace

extern "C" {

const char* miniattn_version(void) { return "miniattn-b200 0.2 sm_100a"; }

// Head dim the kernels are instantiated for.  D = 96 runs on the D = 128 kernels: the tensor maps
// carry the true extent, so TMA zero-fills columns 96..127 of every Q, K and V tile on the way in
// (zeros change neither Q K^T nor P V) and clips them from the O tile on the way out.
static int kernel_head_dim(int D) { return D == 96 ? 128 : D; }

const char* miniattn_last_error_string(void) { return g_err; }

// Shared argument checks of the forward entry points.  Returns 1 when there is nothing to do.
static int check_fwd_params(const MiniAttnFwdParams* p) {
  if (p == nullptr) return fail(MINIATTN_EINVAL, "params is null");
  if (p->dtype != MINIATTN_FP16 && p->dtype != MINIATTN_BF16)
    return fail(MINIATTN_EUNSUPPORTED, "dtype must be fp16 (0) or bf16 (1), got %d", p->dtype);
  if (p->D != 64 && p->D != 96 && p->D != 128)
    return fail(MINIATTN_EUNSUPPORTED, "head dim %d not supported (64, 96 or 128)", p->D);
  if (p->B < 0 || p->Hq < 0 || p->Hkv < 0 || p->Nq < 0 || p->Nk < 0)
    return fail(MINIATTN_EINVAL, "negative size");
  if (p->B == 0 || p->Hq == 0 || p->Nq == 0) return 1;  // empty output: nothing to do
  if (p->Hkv == 0 || p->Hq % p->Hkv != 0)
    return fail(MINIATTN_EINVAL, "Hq (%d) must be a positive multiple of Hkv (%d)", p->Hq, p->Hkv);
  if (p->Hq > 65535 || p->B > 65535)
    return fail(MINIATTN_EUNSUPPORTED, "B and Hq must not exceed 65535");
  if (p->causal != 0 && p->causal != 1) return fail(MINIATTN_EINVAL, "causal must be 0 or 1");
  if (p->kernel < MINIATTN_KERNEL_AUTO || p->kernel > MINIATTN_KERNEL_WS)
    return fail(MINIATTN_EINVAL, "unknown kernel selector %d", p->kernel);
  if ((p->carry_in != 0 && p->carry_in != 1) || (p->carry_out != 0 && p->carry_out != 1))
    return fail(MINIATTN_EINVAL, "carry_in and carry_out must be 0 or 1");
  const bool carry = p->carry_in || p->carry_out;
  if (carry) {
    if (p->carry == nullptr) return fail(MINIATTN_EINVAL, "carry_in / carry_out set but carry is null");
    if (reinterpret_cast<uintptr_t>(p->carry) % 256 != 0)
      return fail(MINIATTN_EINVAL, "carry must be 256-byte aligned");
    if (p->kernel == MINIATTN_KERNEL_SIMPLE)
      return fail(MINIATTN_EUNSUPPORTED, "the carried state needs the warp-specialised kernel");
    const int tiles = (p->Nq + ma::kTileM - 1) / ma::kTileM;
    if (p->carry_tile0 < 0 || p->carry_tiles < 0 ||
        (p->carry_tiles == 0 ? p->carry_tile0 != 0 : p->carry_tile0 + tiles > p->carry_tiles))
      return fail(MINIATTN_EINVAL, "carry_tile0 (%d) + the %d Q tiles of this call exceed carry_tiles (%d)",
                  p->carry_tile0, tiles, p->carry_tiles);
  }
  int rc;
  if ((rc = check_tensor(p->q, p->q_stride, p->D, "q")) != 0) return rc;
  // a call that only stores the running state writes no output: o may be null then
  if (!(p->carry_out && p->o == nullptr) && (rc = check_tensor(p->o, p->o_stride, p->D, "o")) != 0) return rc;
  // With no keys every row is fully masked; K/V pointers are still handed to the tensor-map
  // encoder, so they must be valid whenever Nk > 0.
  const bool has_keys = p->Nk > 0;
  if (has_keys) {
    if ((rc = check_tensor(p->k, p->k_stride, p->D, "k")) != 0) return rc;
    if ((rc = check_tensor(p->v, p->v_stride, p->D, "v")) != 0) return rc;
  }

  return MINIATTN_OK;
}

// Group size of the work-item order (FwdArgs::bh_group).  When the K and V of all heads together
// exceed what L2 keeps of them (its 126 MB are two partitions, and Q and O stream through as well),
// walking all heads at once makes every wave of CTAs fetch K and V from HBM again: measured on a
// 16384 x 16384 task with 32 heads, 7.6 GB of DRAM reads for 0.4 GB of operands.  Groups whose K/V
// fit a share of L2 bring that back to about one read.  A group is a whole number of KV heads
// (with the query heads they serve) and divides B*Hq.
#ifndef MINIATTN_GROUP_TOTAL_MB
#define MINIATTN_GROUP_TOTAL_MB 48
#define MINIATTN_GROUP_SHARE_MB 40
#endif
static int head_group(const MiniAttnFwdParams* p, int pack) {
  const long long bh_total = static_cast<long long>(p->B) * (p->Hq / pack);
  if (p->Hkv <= 0 || p->Hq % p->Hkv != 0) return static_cast<int>(bh_total > 0 ? bh_total : 1);
  const long long g = p->Hq / p->Hkv / pack;                        // work-item heads per KV head
  const long long kv_heads = static_cast<long long>(p->B) * p->Hkv;
  const long long per_kv = 2ll * p->Nk * kernel_head_dim(p->D) * 2; // K and V bytes of one KV head
  if (per_kv * kv_heads < (static_cast<long long>(MINIATTN_GROUP_TOTAL_MB) << 20)) return static_cast<int>(bh_total);
  long long want = (static_cast<long long>(MINIATTN_GROUP_SHARE_MB) << 20) / (per_kv > 0 ? per_kv : 1);
  if (want < 1) want = 1;
  long long d = 1;
  for (long long c = 1; c <= want && c <= kv_heads; ++c)
    if (kv_heads % c == 0) d = c;
  return static_cast<int>(d * g);
}

// K/V tiles that the first n pairs of Q tiles visit together: the sum of kv_tiles_of, in at most 128 steps however
// many pairs there are (one Q tile holds a single token where 128 heads share it).  Pair i ends at key end0 + step * i,
// so pairs 128 apart differ by step tiles exactly.
static long long kv_tiles_of_pairs(const ma::FwdArgs& a, long long n) {
  const long long all = (static_cast<long long>(a.Nk) + ma::kTileN - 1) / ma::kTileN;
  if (!a.causal) return n * all;
  const long long step = 2 * a.tpt, end0 = a.q_pos0 - a.k_pos0 + step;
  auto first_at = [&](long long key) {  // first pair that ends at `key` or later
    return std::clamp<long long>(end0 >= key ? 0 : (key - end0 + step - 1) / step, 0, n);
  };
  const long long lo = first_at(1), hi = first_at(a.Nk);  // pairs before lo see nothing, those from hi on every key
  long long sum = (n - hi) * all;
  for (long long i = lo; i < std::min(lo + ma::kTileN, hi); ++i) {
    const long long times = (hi - i + ma::kTileN - 1) / ma::kTileN;  // pairs i, i + 128, ... before hi
    sum += times * ((end0 + step * i + ma::kTileN - 1) / ma::kTileN) + step * (times * (times - 1) / 2);
  }
  return sum;
}

// Query heads that share a Q tile: all G heads of a KV head, or 1.  Packed, a tile holds 128 / G tokens of
// each head: the tail of a token count that is no multiple of 128 is padded once per KV head instead of once
// per query head, and under a causal mask a pair of tiles spans 256 / G tokens, so that its rows share more
// of their last K/V tiles (N = 1024, G = 4: 4.5 instead of 5 tiles per pair on average).  Taken where that
// saves at least 1 % of the K/V tiles to visit; where G does not divide 128 some rows are lost to padding.
// Measured (one head per tile / packed, causal bf16, D = 128): 777 against 3333 keys, 2 x 24/8 heads 69.0 /
// 62.5 us; N = 4096, 4 x 32/8 heads 500 / 488, 1 x 16/4 heads 58.3 / 56.5; N = 1024, 2 x 16/4 heads 19.1 / 19.1
// (one wave, as long as its longest item).  With nothing to save the packed kernel is 0.3 us slower (two more
// divisions and 5-D copies), so it is not taken then.
static int head_pack(const MiniAttnFwdParams* p) {
  const int g = p->Hkv > 0 ? p->Hq / p->Hkv : 1;
  if (g < 2 || g > ma::kTileM || p->Hq % g != 0 || p->Hq / g != p->Hkv || p->Nq <= 0 || p->Nk <= 0) return 1;
  if (p->kernel == MINIATTN_KERNEL_SIMPLE || p->carry_in || p->carry_out) return 1;
  long long visits[2];
  for (int packed = 0; packed < 2; ++packed) {
    ma::FwdArgs a{};
    a.Nq = p->Nq;
    a.Nk = p->Nk;
    a.causal = p->causal;
    a.q_pos0 = p->q_pos0;
    a.k_pos0 = p->k_pos0;
    a.tpt = ma::kTileM / (packed ? g : 1);
    const int n_tiles = (p->Nq + a.tpt - 1) / a.tpt;
    const int last = (n_tiles - 1) / 2, last_nt = n_tiles - 2 * last;
    // a step of a tile alone takes about two thirds of a pair's (us at D = 64 / 96 / 128: 0.94 and 1.45, 0.94 and 1.49,
    // 0.93 and 1.57)
    visits[packed] = 3 * kv_tiles_of_pairs(a, last) +
                     (last_nt == 2 ? 3 : 2) * static_cast<long long>(ma::kv_tiles_of(a, last * 2 * a.tpt, last_nt));
    if (!packed) visits[0] *= g;
  }
  return visits[1] * 100 <= visits[0] * 99 ? g : 1;
}

static void fill_args(const MiniAttnFwdParams* p, ma::FwdArgs* a, int pack) {
  a->lse = p->lse;
  a->status = p->status;
  a->q_pos0 = p->q_pos0;
  a->k_pos0 = p->k_pos0;
  a->Nq = p->Nq;
  a->Nk = p->Nk;
  a->Hq = p->Hq / pack;
  a->Hkv = p->Hkv;
  a->B = p->B;
  a->causal = p->causal;
  a->d96 = p->D == 96;
  a->scale = p->softmax_scale > 0.f ? p->softmax_scale : 1.0f / sqrtf((float)p->D);
  a->scale_log2 = a->scale * 1.4426950408889634f;
  a->pack = pack;
  a->tpt = ma::kTileM / pack;
  a->n_q_tiles = (p->Nq + a->tpt - 1) / a->tpt;
  a->n_pair_items = 0;  // set by the warp-specialised launcher
  a->bh_group = head_group(p, pack);
  ma::set_divisors(a);
  a->sq = nullptr;
  a->sk = nullptr;
  a->part_o = nullptr;
  a->part_ml = nullptr;
  a->counters = nullptr;
  a->carry_o = nullptr;
  a->carry_ml = nullptr;
  a->carry_mode = 0;
  a->carry_tile0 = 0;
  a->carry_tiles = 0;
}

static int check_device(int* sms) {
  int major = 0, rc;
  if ((rc = device_sm_count(sms, &major)) != 0) return rc;
  if (major != 10)
    return fail(MINIATTN_EUNSUPPORTED,
                "this library holds sm_100a code only; current device has compute capability %d.x",
                major);
  return MINIATTN_OK;
}

// Plans of recent shapes (planning costs up to a few milliseconds of host time; launches of one shape repeat).
// A plan depends on the sizes only through the K/V tiles that each pair of Q tiles visits, so a call whose sizes
// are new is looked up a second time by those: while a context grows a token at a time, 128 calls share a plan.
// Guarded by a mutex; what is handed out is shared and never changed.
namespace {
struct PlanKey {
  int Nq, Nk, B, Hq, causal, D, sms, group, pack;
  long long diag;
  bool operator==(const PlanKey& o) const {
    return Nq == o.Nq && Nk == o.Nk && B == o.B && Hq == o.Hq && causal == o.causal && D == o.D &&
           sms == o.sms && group == o.group && pack == o.pack && diag == o.diag;
  }
};
struct PlanSlot {
  PlanKey key;              // the sizes it was last used for
  std::vector<int> tiles;   // of each pair
  std::shared_ptr<const ma::FwdPlan> plan;
  bool serves(const PlanKey& k, const std::vector<int>& t) const {
    return static_cast<long long>(key.B) * key.Hq == static_cast<long long>(k.B) * k.Hq && key.D == k.D &&
           key.sms == k.sms && key.group == k.group && tiles == t;
  }
};
constexpr size_t kPlanSlots = 64;
std::shared_ptr<const ma::FwdPlan> cached_plan(const ma::FwdArgs& a, int D, int sms) {
  static std::mutex mu;
  static std::vector<PlanSlot> cache;
  static size_t next = 0;
  static const auto never_cut = std::make_shared<const ma::FwdPlan>(ma::FwdPlan{});
  if (!ma::plan_considered(a, sms)) return never_cut;
  const PlanKey key{a.Nq, a.Nk, a.B, a.Hq, a.causal, D, sms, a.bh_group, a.pack, a.causal ? a.q_pos0 - a.k_pos0 : 0};
  {
    std::lock_guard<std::mutex> g(mu);
    for (const PlanSlot& s : cache)
      if (s.key == key) return s.plan;
  }
  std::vector<int> tiles((a.n_q_tiles + 1) / 2);
  for (size_t i = 0; i < tiles.size(); ++i) {
    const int q0 = static_cast<int>(i) * 2 * a.tpt;
    tiles[i] = ma::kv_tiles_of(a, q0, q0 + a.tpt < a.Nq ? 2 : 1);
  }
  {
    std::lock_guard<std::mutex> g(mu);
    for (PlanSlot& s : cache)
      if (s.serves(key, tiles)) {
        s.key = key;
        return s.plan;
      }
  }
  auto plan = std::make_shared<ma::FwdPlan>();
  ma::plan_fwd(a, D, sms, plan.get());
  std::lock_guard<std::mutex> g(mu);
  PlanSlot slot{key, std::move(tiles), plan};
  if (cache.size() < kPlanSlots) cache.push_back(std::move(slot));
  else cache[next++ % kPlanSlots] = std::move(slot);
  return plan;
}

constexpr size_t kCounterBytes = 16384;  // (arrived, published) x 2 Q tiles x kPlanCap cut items, rounded up
static_assert(4 * ma::kPlanCap * sizeof(int) <= kCounterBytes, "counter region too small");
size_t align256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }
size_t scratch_bytes_of(const ma::FwdPlan& plan, int D) {
  if (!plan.split) return 0;
  const size_t rows = static_cast<size_t>(plan.n_slots) * 2 * ma::kTileM;
  return kCounterBytes + align256(rows * sizeof(float2)) + rows * D * sizeof(float);
}
}  // namespace

// Points the kernel arguments at the three regions of a balanced launch's scratch.
static int bind_scratch(const ma::FwdPlan& plan, int D, void* scratch, size_t scratch_bytes, ma::FwdArgs* a) {
  const size_t need = scratch_bytes_of(plan, D);
  if (scratch_bytes < need)
    return fail(MINIATTN_EINVAL, "scratch holds %zu bytes, this launch needs %zu "
                "(miniattn_fwd_balanced_scratch_bytes)", scratch_bytes, need);
  if (reinterpret_cast<uintptr_t>(scratch) % 256 != 0)
    return fail(MINIATTN_EINVAL, "scratch must be 256-byte aligned");
  uint8_t* base = static_cast<uint8_t*>(scratch);
  const size_t rows = static_cast<size_t>(plan.n_slots) * 2 * ma::kTileM;
  a->counters = reinterpret_cast<int*>(base);
  a->part_ml = reinterpret_cast<float2*>(base + kCounterBytes);
  a->part_o = reinterpret_cast<float*>(base + kCounterBytes + align256(rows * sizeof(float2)));
  return MINIATTN_OK;
}

// ---- calls with few query rows per KV head (fwd_decode.cu) ----
static void decode_plan_of(const MiniAttnFwdParams* p, int sms, bool cut, ma::DecodePlan* d) {
  *d = ma::DecodePlan{};
  if (p->kernel != MINIATTN_KERNEL_AUTO || p->carry_in || p->carry_out) return;
  if (p->B <= 0 || p->Hkv <= 0 || p->Hq <= 0 || p->Hq % p->Hkv != 0 || p->Nq <= 0 || p->Nk <= 0) return;
  ma::plan_decode(p->B, p->Hq, p->Hkv, p->Nq, p->Nk, kernel_head_dim(p->D), p->causal, p->q_pos0 - p->k_pos0, sms, cut, d);
}

static size_t decode_scratch_bytes(const ma::DecodePlan& d, int D) {
  if (d.rg == 0 || d.total / d.tiles == d.n_ctas) return 0;  // one whole item per CTA: nothing is cut
  const size_t rows = static_cast<size_t>(2 * d.n_ctas) * 16 * d.rg;
  return kCounterBytes + align256(rows * sizeof(float2)) + rows * kernel_head_dim(D) * sizeof(float);
}

// scratch: decode_scratch_bytes(d, p->D) bytes, 256-byte aligned; null where that is 0.
static int fwd_decode(const MiniAttnFwdParams* p, const ma::DecodePlan& d, void* scratch, cudaStream_t st) {
  const CUtensorMapDataType dt =
      p->dtype == MINIATTN_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUtensorMap tm[2];
  int rc;
  if ((rc = make_map(&tm[0], p->k, 2, dt, p->D, p->Nk, p->Hkv, p->B, p->k_stride, ma::kBoxCols, 64, "k")) != 0)
    return rc;
  if ((rc = make_map(&tm[1], p->v, 2, dt, p->D, p->Nk, p->Hkv, p->B, p->v_stride, ma::kBoxCols, 64, "v")) != 0)
    return rc;
  ma::DecodeArgs a{};
  a.q = static_cast<const uint16_t*>(p->q);
  a.o = static_cast<uint16_t*>(p->o);
  for (int i = 0; i < 3; ++i) {
    a.qs[i] = p->q_stride[i];
    a.os[i] = p->o_stride[i];
  }
  a.lse = p->lse;
  a.status = p->status;
  a.diag = p->q_pos0 - p->k_pos0;
  a.total = d.total;
  a.Nq = p->Nq;
  a.Nk = p->Nk;
  a.Hq = p->Hq;
  a.Hkv = p->Hkv;
  a.G = p->Hq / p->Hkv;
  a.D = p->D;
  a.causal = p->causal;
  a.rows = a.G * p->Nq;
  a.n_rb = d.n_rb;
  a.tiles = d.tiles;
  a.small = (d.n_ctas + 1ll) <= 0x7fffffffll / d.total;
  a.by_ctas = ma::fast_div(d.n_ctas);
  a.by_tiles = ma::fast_div(d.tiles);
  a.by_total = ma::fast_div(a.small ? static_cast<uint32_t>(d.total) : 1u);
  a.by_rb = ma::fast_div(d.n_rb);
  a.by_hkv = ma::fast_div(p->Hkv);
  a.by_g = ma::fast_div(a.G);
  a.scale_log2 = (p->softmax_scale > 0.f ? p->softmax_scale : 1.0f / sqrtf((float)p->D)) * 1.4426950408889634f;
  if (scratch != nullptr) {
    uint8_t* base = static_cast<uint8_t*>(scratch);
    const size_t rows = static_cast<size_t>(2 * d.n_ctas) * 16 * d.rg;
    a.counters = reinterpret_cast<int*>(base);
    a.part_ml = reinterpret_cast<float2*>(base + kCounterBytes);
    a.part_o = reinterpret_cast<float*>(base + kCounterBytes + align256(rows * sizeof(float2)));
  }
  const cudaError_t e =
      ma::launch_fwd_decode(kernel_head_dim(p->D), p->dtype == MINIATTN_BF16, tm, a, d.rg, d.n_ctas, st);
  if (e != cudaSuccess) return fail(MINIATTN_ECUDA, "kernel launch failed: %s", cudaGetErrorString(e));
  return MINIATTN_OK;
}

// Forward launch shared by miniattn_fwd and miniattn_fwd_balanced (scratch == nullptr: plain).
static int fwd_common(const MiniAttnFwdParams* p, void* scratch, size_t scratch_bytes, void* stream) {
  g_err[0] = 0;
  int rc = check_fwd_params(p);
  if (rc != 0) return rc > 0 ? MINIATTN_OK : rc;
  const bool has_keys = p->Nk > 0;
  int sms = 0;
  if ((rc = check_device(&sms)) != 0) return rc;
  ma::DecodePlan dec;
  decode_plan_of(p, sms, scratch != nullptr, &dec);
  // Scratch that does not hold the pieces of the few-rows kernel may still do for the general one, which often
  // needs none (a caller may have sized it by miniattn_plan_fwd): the call runs there, or is refused there.
  const size_t dec_need = decode_scratch_bytes(dec, p->D);
  if (dec.rg != 0 && (dec_need == 0 || (scratch_bytes >= dec_need && reinterpret_cast<uintptr_t>(scratch) % 256 == 0)))
    return fwd_decode(p, dec, dec_need > 0 ? scratch : nullptr, reinterpret_cast<cudaStream_t>(stream));

  const CUtensorMapDataType dt =
      p->dtype == MINIATTN_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUtensorMap tm[4];
  const bool simple = p->kernel == MINIATTN_KERNEL_SIMPLE;
  ma::FwdArgs a;
  fill_args(p, &a, head_pack(p));
  // rows: of the box, a whole tile or what one warp stores of it
  auto q_map = [&](CUtensorMap* out, const void* base, const int64_t stride[3], int rows, const char* what) {
    return a.pack == 1 ? make_map(out, base, 2, dt, p->D, p->Nq, p->Hq, p->B, stride, ma::kBoxCols, rows, what)
                       : make_map_packed(out, base, dt, p->D, p->Nq, a.Hq, p->B, stride, a.pack, rows / a.pack, what);
  };
  if ((rc = q_map(&tm[0], p->q, p->q_stride, ma::kTileM, "q")) != 0) return rc;
  if (has_keys) {
    if ((rc = make_map(&tm[1], p->k, 2, dt, p->D, p->Nk, p->Hkv, p->B, p->k_stride, ma::kBoxCols,
                       ma::kTileN, "k")) != 0)
      return rc;
    if ((rc = make_map(&tm[2], p->v, 2, dt, p->D, p->Nk, p->Hkv, p->B, p->v_stride, ma::kBoxCols,
                       ma::kTileN, "v")) != 0)
      return rc;
  } else {
    tm[1] = tm[0];
    tm[2] = tm[0];
  }
  if (p->o == nullptr) {
    tm[3] = tm[0];  // state-only call: the kernel never stores through the output map
  } else if ((rc = q_map(&tm[3], p->o, p->o_stride,
                         simple || ma::kWarpRows % a.pack != 0 ? ma::kTileM : ma::kWarpRows, "o")) != 0) {
    return rc;
  }

  const int kd = kernel_head_dim(p->D);
  const bool carry = p->carry_in || p->carry_out;
  if (carry) {
    a.carry_tiles = p->carry_tiles > 0 ? p->carry_tiles : a.n_q_tiles;
    a.carry_tile0 = p->carry_tile0;
    const size_t rows = static_cast<size_t>(p->B) * p->Hq * a.carry_tiles * ma::kTileM;
    a.carry_o = static_cast<float*>(p->carry);
    a.carry_ml = reinterpret_cast<float2*>(static_cast<uint8_t*>(p->carry) + rows * kd * sizeof(float));
    a.carry_mode = (p->carry_in ? 1 : 0) | (p->carry_out ? 2 : 0);
  }

  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  cudaError_t e;
  if (simple) {
    e = ma::launch_fwd_simple(kd, p->dtype == MINIATTN_BF16, tm, a, st);
  } else {
    // a call that carries ring state always takes the plain launch
    std::shared_ptr<const ma::FwdPlan> plan;
    if (scratch != nullptr && has_keys && !carry) plan = cached_plan(a, kd, sms);
    if (plan && plan->split) {
      if ((rc = bind_scratch(*plan, kd, scratch, scratch_bytes, &a)) != 0) return rc;
      e = ma::launch_fwd_ws_plan(kd, p->dtype == MINIATTN_BF16, false, tm, a, *plan, st);
    } else {
      e = ma::launch_fwd_ws(kd, p->dtype == MINIATTN_BF16, tm, a, sms, st);
    }
  }
  if (e != cudaSuccess)
    return fail(MINIATTN_ECUDA, "kernel launch failed: %s", cudaGetErrorString(e));
  return MINIATTN_OK;
}

int miniattn_fwd(const MiniAttnFwdParams* p, void* stream) { return fwd_common(p, nullptr, 0, stream); }

int miniattn_fwd_balanced(const MiniAttnFwdParams* p, void* scratch, size_t scratch_bytes, void* stream) {
  if (scratch == nullptr && scratch_bytes != 0) {
    g_err[0] = 0;
    return fail(MINIATTN_EINVAL, "scratch is null but scratch_bytes is %zu", scratch_bytes);
  }
  return fwd_common(p, scratch, scratch_bytes, stream);
}

static int check_plan_params(const MiniAttnFwdParams* p, int sm_count, int* sms) {
  if (p == nullptr) return fail(MINIATTN_EINVAL, "params is null");
  if (p->D != 64 && p->D != 96 && p->D != 128)
    return fail(MINIATTN_EUNSUPPORTED, "head dim %d not supported (64, 96 or 128)", p->D);
  if (p->B < 0 || p->Hq < 0 || p->Nq < 0 || p->Nk < 0) return fail(MINIATTN_EINVAL, "negative size");
  if (p->Hq > 65535 || p->B > 65535)
    return fail(MINIATTN_EUNSUPPORTED, "B and Hq must not exceed 65535");
  *sms = sm_count;
  return sm_count > 0 ? MINIATTN_OK : check_device(sms);
}

// Plan of a forward launch for `sm_count` SMs (<= 0: the current device's).  Host arithmetic only.
static int plan_info_of(const MiniAttnFwdParams* p, bool may_pack, int sm_count, MiniAttnPlanInfo* info,
                        MiniAttnPlanPiece* pieces, int32_t cap) {
  g_err[0] = 0;
  if (info == nullptr) return fail(MINIATTN_EINVAL, "info is null");
  memset(info, 0, sizeof(*info));
  int sms = 0, rc;
  if ((rc = check_plan_params(p, sm_count, &sms)) != 0) return rc;
  ma::FwdArgs a;
  fill_args(p, &a, may_pack ? head_pack(p) : 1);
  const long long n_items = static_cast<long long>((a.n_q_tiles + 1) / 2) * a.Hq * p->B;
  info->sm_count = sms;
  info->n_ctas = n_items;
  info->head_group = a.bh_group;
  if (p->B == 0 || p->Hq == 0 || p->Nq == 0 || p->Nk == 0 ||
      (p->kernel != MINIATTN_KERNEL_AUTO && p->kernel != MINIATTN_KERNEL_WS) || p->carry_in || p->carry_out)
    return MINIATTN_OK;
  const int kd = kernel_head_dim(p->D);
  std::shared_ptr<const ma::FwdPlan> plan = cached_plan(a, kd, sms);
  info->est_plain = plan->est_plain;
  info->est_balanced = plan->est_balanced;
  if (!plan->split) return MINIATTN_OK;
  info->split = 1;
  info->n_whole = plan->n_whole;
  info->n_pieces = plan->n_table;
  info->n_ctas = plan->n_whole + plan->n_table;
  info->n_cut_items = plan->n_cut_items;
  info->n_slots = plan->n_slots;
  info->scratch_bytes = static_cast<int64_t>(scratch_bytes_of(*plan, kd));
  if (pieces != nullptr)
    for (int k = 0; k < plan->n_table && k < cap; ++k) {
      const ma::PlanEntry& e = plan->table.e[k];
      pieces[k].item = static_cast<int32_t>(e.item);
      pieces[k].t0 = e.t0;
      pieces[k].t1 = e.t1;
      pieces[k].part = e.part;
      pieces[k].nparts = e.nparts;
      pieces[k].slot = e.nparts > 1 ? e.slot0 + e.part : -1;
    }
  return MINIATTN_OK;
}

int miniattn_plan_fwd(const MiniAttnFwdParams* p, int sm_count, MiniAttnPlanInfo* info,
                      MiniAttnPlanPiece* pieces, int32_t cap) {
  return plan_info_of(p, true, sm_count, info, pieces, cap);
}

int64_t miniattn_fwd_carry_bytes(const MiniAttnFwdParams* p) {
  g_err[0] = 0;
  if (p == nullptr) return fail(MINIATTN_EINVAL, "params is null");
  if (p->D != 64 && p->D != 96 && p->D != 128)
    return fail(MINIATTN_EUNSUPPORTED, "head dim %d not supported (64, 96 or 128)", p->D);
  if (p->B < 0 || p->Hq < 0 || p->Nq < 0) return fail(MINIATTN_EINVAL, "negative size");
  const int64_t tiles = static_cast<int64_t>(p->B) * p->Hq * ((p->Nq + ma::kTileM - 1) / ma::kTileM);
  return tiles * ma::kTileM * (kernel_head_dim(p->D) * 4 + 8);
}

int64_t miniattn_fwd_scratch_bytes(const MiniAttnFwdParams* p, int32_t int8qk, int sm_count) {
  g_err[0] = 0;
  int sms = 0, rc;
  if ((rc = check_plan_params(p, sm_count, &sms)) != 0) return rc;
  if (!int8qk) {  // a call for the few-rows kernel needs no plan of the general one: a decode loop never makes any
    ma::DecodePlan dec;
    decode_plan_of(p, sms, true, &dec);
    if (dec.rg != 0) return static_cast<int64_t>(decode_scratch_bytes(dec, p->D));
  }
  MiniAttnPlanInfo info;
  if ((rc = plan_info_of(p, !int8qk, sms, &info, nullptr, 0)) != 0) return rc;  // INT8-QK does not pack heads
  return info.scratch_bytes;
}

int64_t miniattn_fwd_balanced_scratch_bytes(const MiniAttnFwdParams* p) {
  const int64_t plain = miniattn_fwd_scratch_bytes(p, 0, 0);
  if (plain < 0 || p->D == 96) return plain;
  const int64_t int8 = miniattn_fwd_scratch_bytes(p, 1, 0);
  return int8 < 0 ? int8 : std::max(plain, int8);
}

static int check_int8_params(const MiniAttnInt8Params* p, bool need_v) {
  if (p == nullptr) return fail(MINIATTN_EINVAL, "params is null");
  MiniAttnFwdParams f = p->fwd;
  if (!need_v) {  // the pre-pass reads q and k only
    f.v = f.k;
    for (int i = 0; i < 3; ++i) f.v_stride[i] = f.k_stride[i];
    if (f.o == nullptr) {
      f.o = const_cast<void*>(f.q);
      for (int i = 0; i < 3; ++i) f.o_stride[i] = f.q_stride[i];
    }
  }
  int rc = check_fwd_params(&f);
  if (rc != 0) return rc;
  if (p->fwd.D == 96) return fail(MINIATTN_EUNSUPPORTED, "the INT8-QK variant takes head dim 64 or 128");
  if (p->fwd.carry_in || p->fwd.carry_out)
    return fail(MINIATTN_EUNSUPPORTED, "the INT8-QK variant does not carry ring state");
  if (p->fwd.Nk == 0) return fail(MINIATTN_EINVAL, "the INT8-QK variant needs at least one key");
  if (!p->q8 || !p->k8 || !p->q_scale || !p->k_scale)
    return fail(MINIATTN_EINVAL, "q8, k8, q_scale and k_scale must not be null");
  if (reinterpret_cast<uintptr_t>(p->q8) % 16 || reinterpret_cast<uintptr_t>(p->k8) % 16)
    return fail(MINIATTN_EINVAL, "q8 and k8 must be 16-byte aligned");
  return MINIATTN_OK;
}

int miniattn_quant_qk_int8(const MiniAttnInt8Params* p, void* stream) {
  g_err[0] = 0;
  int rc = check_int8_params(p, false);
  if (rc != 0) return rc > 0 ? MINIATTN_OK : rc;
  if (!p->k_partial) return fail(MINIATTN_EINVAL, "k_partial scratch must not be null");
  int sms = 0;
  if ((rc = check_device(&sms)) != 0) return rc;
  const MiniAttnFwdParams& f = p->fwd;
  const float scale = f.softmax_scale > 0.f ? f.softmax_scale : 1.0f / sqrtf((float)f.D);
  const long long qs[3] = {f.q_stride[0], f.q_stride[1], f.q_stride[2]};
  const long long ks[3] = {f.k_stride[0], f.k_stride[1], f.k_stride[2]};
  cudaError_t e = ma::launch_quant_qk(f.D, f.dtype == MINIATTN_BF16, f.q, qs, f.k, ks, f.B, f.Hq, f.Hkv,
                                      f.Nq, f.Nk, scale * 1.4426950408889634f, p->q8, p->k8, p->q_scale,
                                      p->k_scale, p->k_partial, p->k_mean,
                                      reinterpret_cast<cudaStream_t>(stream));
  if (e != cudaSuccess)
    return fail(MINIATTN_ECUDA, "kernel launch failed: %s", cudaGetErrorString(e));
  return MINIATTN_OK;
}

int miniattn_quant_qk_int8_static(const MiniAttnInt8Params* p, void* stream) {
  g_err[0] = 0;
  int rc = check_int8_params(p, false);
  if (rc != 0) return rc > 0 ? MINIATTN_OK : rc;
  int sms = 0;
  if ((rc = check_device(&sms)) != 0) return rc;
  const MiniAttnFwdParams& f = p->fwd;
  const long long need = (long long)f.B * f.Hkv * ((f.Nk + 1023) / 1024) * f.D;
  if (need > ma::static_colsum_capacity())
    return fail(MINIATTN_EUNSUPPORTED,
                "B*Hkv*ceil(Nk/1024)*D = %lld floats of column-sum scratch exceed the built-in %lld; "
                "use miniattn_quant_qk_int8 with a caller-provided k_partial buffer",
                need, ma::static_colsum_capacity());
  const float scale = f.softmax_scale > 0.f ? f.softmax_scale : 1.0f / sqrtf((float)f.D);
  const long long qs[3] = {f.q_stride[0], f.q_stride[1], f.q_stride[2]};
  const long long ks[3] = {f.k_stride[0], f.k_stride[1], f.k_stride[2]};
  cudaError_t e = ma::launch_quant_qk_static(f.D, f.dtype == MINIATTN_BF16, f.q, qs, f.k, ks, f.B, f.Hq,
                                             f.Hkv, f.Nq, f.Nk, scale * 1.4426950408889634f, p->q8, p->k8,
                                             p->q_scale, p->k_scale, p->k_mean,
                                             reinterpret_cast<cudaStream_t>(stream));
  if (e != cudaSuccess)
    return fail(MINIATTN_ECUDA, "pre-pass set-up or launch failed: %s", cudaGetErrorString(e));
  return MINIATTN_OK;
}

static int int8_common(const MiniAttnInt8Params* p, void* scratch, size_t scratch_bytes, void* stream) {
  g_err[0] = 0;
  int rc = check_int8_params(p, true);
  if (rc != 0) return rc > 0 ? MINIATTN_OK : rc;
  int sms = 0;
  if ((rc = check_device(&sms)) != 0) return rc;
  const MiniAttnFwdParams& f = p->fwd;
  const CUtensorMapDataType dt =
      f.dtype == MINIATTN_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  // int8 rows are D bytes wide: one box per tile, 64-byte swizzle at D=64, 128-byte at D=128
  const CUtensorMapSwizzle sw8 = f.D == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B;
  const int64_t q8s[3] = {(int64_t)f.Hq * f.Nq * f.D, (int64_t)f.Nq * f.D, f.D};
  const int64_t k8s[3] = {(int64_t)f.Hkv * f.Nk * f.D, (int64_t)f.Nk * f.D, f.D};
  CUtensorMap tm[4];
  if ((rc = make_map(&tm[0], p->q8, 1, CU_TENSOR_MAP_DATA_TYPE_UINT8, f.D, f.Nq, f.Hq, f.B, q8s, f.D,
                     ma::kTileM, "q8", sw8)) != 0)
    return rc;
  if ((rc = make_map(&tm[1], p->k8, 1, CU_TENSOR_MAP_DATA_TYPE_UINT8, f.D, f.Nk, f.Hkv, f.B, k8s, f.D,
                     ma::kTileN, "k8", sw8)) != 0)
    return rc;
  if ((rc = make_map(&tm[2], f.v, 2, dt, f.D, f.Nk, f.Hkv, f.B, f.v_stride, ma::kBoxCols, ma::kTileN,
                     "v")) != 0)
    return rc;
  if ((rc = make_map(&tm[3], f.o, 2, dt, f.D, f.Nq, f.Hq, f.B, f.o_stride, ma::kBoxCols, ma::kWarpRows,
                     "o")) != 0)
    return rc;
  ma::FwdArgs a;
  fill_args(&f, &a, 1);
  a.sq = p->q_scale;
  a.sk = p->k_scale;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  cudaError_t e;
  std::shared_ptr<const ma::FwdPlan> plan;
  if (scratch != nullptr) plan = cached_plan(a, f.D, sms);
  if (plan && plan->split) {
    if ((rc = bind_scratch(*plan, f.D, scratch, scratch_bytes, &a)) != 0) return rc;
    e = ma::launch_fwd_ws_plan(f.D, f.dtype == MINIATTN_BF16, true, tm, a, *plan, st);
  } else {
    e = ma::launch_fwd_ws_int8qk(f.D, f.dtype == MINIATTN_BF16, tm, a, sms, st);
  }
  if (e != cudaSuccess)
    return fail(MINIATTN_ECUDA, "kernel launch failed: %s", cudaGetErrorString(e));
  return MINIATTN_OK;
}

int miniattn_fwd_int8qk(const MiniAttnInt8Params* p, void* stream) { return int8_common(p, nullptr, 0, stream); }

int miniattn_fwd_int8qk_balanced(const MiniAttnInt8Params* p, void* scratch, size_t scratch_bytes, void* stream) {
  if (scratch == nullptr && scratch_bytes != 0) {
    g_err[0] = 0;
    return fail(MINIATTN_EINVAL, "scratch is null but scratch_bytes is %zu", scratch_bytes);
  }
  return int8_common(p, scratch, scratch_bytes, stream);
}

int miniattn_merge_partials(const MiniAttnMergeParams* p, void* stream) {
  g_err[0] = 0;
  if (p == nullptr) return fail(MINIATTN_EINVAL, "params is null");
  if (p->rows < 0) return fail(MINIATTN_EINVAL, "negative row count");
  if (p->D != 64 && p->D != 128)
    return fail(MINIATTN_EUNSUPPORTED, "head dim %d not supported (64 or 128)", p->D);
  if (p->dtype != MINIATTN_FP16 && p->dtype != MINIATTN_BF16)
    return fail(MINIATTN_EUNSUPPORTED, "dtype must be fp16 (0) or bf16 (1), got %d", p->dtype);
  if (p->init != 0 && p->init != 1) return fail(MINIATTN_EINVAL, "init must be 0 or 1");
  if (p->rows == 0) return MINIATTN_OK;
  if (!p->acc_o || !p->acc_lse || !p->part_o || !p->part_lse)
    return fail(MINIATTN_EINVAL, "acc_o, acc_lse, part_o and part_lse must not be null");
  if (reinterpret_cast<uintptr_t>(p->acc_o) % 16 || reinterpret_cast<uintptr_t>(p->part_o) % 16 ||
      (p->out && reinterpret_cast<uintptr_t>(p->out) % 16))
    return fail(MINIATTN_EINVAL, "acc_o, part_o and out must be 16-byte aligned");
  int sms = 0, rc;
  if ((rc = check_device(&sms)) != 0) return rc;
  long long rows_per_slab = p->rows, slab_stride = p->rows * p->D;
  if (p->out_rows_per_slab > 0) {
    if (p->rows % p->out_rows_per_slab != 0)
      return fail(MINIATTN_EINVAL, "rows must be a multiple of out_rows_per_slab");
    if (p->out_slab_stride < p->out_rows_per_slab * p->D || p->out_slab_stride % 8 != 0)
      return fail(MINIATTN_EINVAL, "out_slab_stride must be a multiple of 8 elements and cover a slab");
    rows_per_slab = p->out_rows_per_slab;
    slab_stride = p->out_slab_stride;
  }
  cudaError_t e = ma::launch_merge_partials(p->acc_o, p->acc_lse, p->part_o, p->part_lse, p->out,
                                            p->rows, p->D, p->dtype == MINIATTN_BF16, p->init,
                                            rows_per_slab, slab_stride, sms,
                                            reinterpret_cast<cudaStream_t>(stream));
  if (e != cudaSuccess)
    return fail(MINIATTN_ECUDA, "kernel launch failed: %s", cudaGetErrorString(e));
  return MINIATTN_OK;
}

static int check_rows(const void* p, int64_t ld, int cols, const char* name) {
  if (p == nullptr) return fail(MINIATTN_EINVAL, "%s is null", name);
  if (reinterpret_cast<uintptr_t>(p) % 16 != 0) return fail(MINIATTN_EINVAL, "%s must be 16-byte aligned", name);
  if (ld % 8 != 0 || ld < cols)
    return fail(MINIATTN_EINVAL, "row stride of %s (%lld) must be a multiple of 8 and cover its %d columns", name,
                (long long)ld, cols);
  return MINIATTN_OK;
}

int miniattn_linear(const MiniAttnLinearParams* p, void* stream) {
  g_err[0] = 0;
  if (p == nullptr) return fail(MINIATTN_EINVAL, "params is null");
  if (p->dtype != MINIATTN_FP16 && p->dtype != MINIATTN_BF16)
    return fail(MINIATTN_EUNSUPPORTED, "dtype must be fp16 (0) or bf16 (1), got %d", p->dtype);
  if (p->n_out < 1 || p->n_out > ma::kLinearMax)
    return fail(MINIATTN_EINVAL, "1 to %d weights, got %d", ma::kLinearMax, p->n_out);
  if (p->M < 0 || p->K <= 0 || p->K % 8 != 0)
    return fail(MINIATTN_EINVAL, "M (%d) must not be negative, K (%d) a positive multiple of 8", p->M, p->K);
  if (p->M == 0) return MINIATTN_OK;
  int rc, N[ma::kLinearMax];
  if ((rc = check_rows(p->x, p->ldx, p->K, "x")) != 0) return rc;
  for (int i = 0; i < p->n_out; ++i) {
    const MiniAttnLinearOut& o = p->out[i];
    if (o.N <= 0 || o.N % 8 != 0) return fail(MINIATTN_EINVAL, "N (%d) must be a positive multiple of 8", o.N);
    if (o.N > ma::kLinearMaxN) return fail(MINIATTN_EUNSUPPORTED, "N (%d) must be at most %d", o.N, ma::kLinearMaxN);
    if ((rc = check_rows(o.w, o.ldw, p->K, "w")) != 0 || (rc = check_rows(o.y, o.ldy, o.N, "y")) != 0) return rc;
    if (o.bias != nullptr && reinterpret_cast<uintptr_t>(o.bias) % 2 != 0)
      return fail(MINIATTN_EINVAL, "bias must be 2-byte aligned");
    N[i] = o.N;
  }
  int sms = 0;
  if ((rc = check_device(&sms)) != 0) return rc;
  const CUtensorMapDataType dt =
      p->dtype == MINIATTN_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  ma::LinearArgs a{};
  bool pays = false;
  a.bn = ma::linear_tile(p->M, p->K, p->n_out, N, sms / 2, &pays);
  if (p->only_if_faster && !pays) return 1;
  a.status = p->status;
  a.M = p->M;
  a.K = p->K;
  a.n_seg = p->n_out;
  if ((rc = make_map_2d(&a.tm_x, p->x, dt, p->M, p->K, p->ldx, 128, 64, CU_TENSOR_MAP_SWIZZLE_128B, "x")) != 0) return rc;
  long long tiles = 0;
  for (int i = 0; i < p->n_out; ++i) {
    const MiniAttnLinearOut& o = p->out[i];
    ma::LinearSeg& s = a.seg[i];
    if ((rc = make_map_2d(&s.tm_w, o.w, dt, o.N, p->K, o.ldw, a.bn / 2, 64, CU_TENSOR_MAP_SWIZZLE_128B, "w")) != 0 ||
        (rc = make_map_2d(&s.tm_y, o.y, dt, p->M, o.N, o.ldy, 32, 16, CU_TENSOR_MAP_SWIZZLE_NONE, "y")) != 0)
      return rc;
    s.bias = static_cast<const uint16_t*>(o.bias);
    s.N = o.N;
    s.bias_16 = reinterpret_cast<uintptr_t>(o.bias) % 16 == 0;
    a.first_tile[i] = static_cast<int>(tiles);
    tiles += (o.N + (a.bn - 1ll)) / a.bn;
  }
  const long long m_tiles = (p->M + 255ll) / 256;
  if (tiles * m_tiles > 0x3fffffffll) return fail(MINIATTN_EUNSUPPORTED, "too many tiles");
  a.by_m_tiles = ma::fast_div(static_cast<uint32_t>(m_tiles));
  a.n_tiles = static_cast<int>(tiles * m_tiles);
  const cudaError_t e =
      ma::launch_linear(p->dtype == MINIATTN_BF16, a, sms / 2, reinterpret_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return fail(MINIATTN_ECUDA, "kernel launch failed: %s", cudaGetErrorString(e));
  return MINIATTN_OK;
}

int miniattn_check_status(int32_t status_word) {
  g_err[0] = 0;
  if (status_word == 0) return MINIATTN_OK;
  static const char* const names[] = {"K/V or Q tile load", "S = QK^T", "O += PV", "P hand-off", "ring slot release",
                                      "(bit 5, not in use)", "partial of another CTA of a cut item"};
  char list[256] = "";
  for (int bit = 0; bit < 7; ++bit)
    if (status_word & (1 << bit)) {
      if (list[0]) strncat(list, ", ", sizeof(list) - strlen(list) - 1);
      strncat(list, names[bit], sizeof(list) - strlen(list) - 1);
    }
  if (status_word & (1 << 30)) {
    if (list[0]) strncat(list, ", ", sizeof(list) - strlen(list) - 1);
    strncat(list, "self-test wait", sizeof(list) - strlen(list) - 1);
  }
  return fail(MINIATTN_EDEVICE_WAIT, "bounded device waits ran out (status word 0x%x): %s", status_word, list);
}

int miniattn_stream_capture_id(void* stream, uint64_t* id) {
  g_err[0] = 0;
  if (id == nullptr) return fail(MINIATTN_EINVAL, "id is null");
  *id = 0;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long n = 0;
  const cudaError_t e = cudaStreamGetCaptureInfo(reinterpret_cast<cudaStream_t>(stream), &status, &n);
  if (e != cudaSuccess) return fail(MINIATTN_ECUDA, "cudaStreamGetCaptureInfo: %s", cudaGetErrorString(e));
  if (status != cudaStreamCaptureStatusNone) *id = n;
  return MINIATTN_OK;
}

int miniattn_selftest_wait(int32_t* status, uint64_t limit_ns, void* stream) {
  g_err[0] = 0;
  if (status == nullptr) return fail(MINIATTN_EINVAL, "status is null");
  if (limit_ns == 0 || limit_ns > 2000000000ull)
    return fail(MINIATTN_EINVAL, "limit_ns must be in (0, 2e9]");
  cudaError_t e = ma::launch_wait_selftest(status, limit_ns, reinterpret_cast<cudaStream_t>(stream));
  if (e != cudaSuccess)
    return fail(MINIATTN_ECUDA, "kernel launch failed: %s", cudaGetErrorString(e));
  return MINIATTN_OK;
}

}  // extern "C"
