// C ABI of the NVFP4 attention forward (see include/fa4_nvfp4.h): argument validation, TMA
// tensor maps, launch configuration.  Host code only; the kernels live in the .cuh files.
#include "../../include/fa4_nvfp4.h"

#include "attn_common.cuh"
#include "attn_ws.cuh"
#include "attn_ws64.cuh"
#include "attn_decode.cuh"
#include "aux_kernels.cuh"
#include "quantize.cuh"

#include <cudaTypedefs.h>
#include <algorithm>
#include <atomic>
#include <map>
#include <mutex>
#include <utility>

namespace {

using namespace fa4;

constexpr uint64_t kDefaultBudgetNs = 2000ull * 1000 * 1000;
// SMs of a B200, for rules that must give one answer on the host alone (the size of a workspace is asked for
// without a device) and for the shares of the streaming kernels; persistent grids ask the device.
constexpr int64_t kSms = 148;

PFN_cuTensorMapEncodeTiled_v12000 get_encode() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) ==
            cudaSuccess &&
        qres == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
    }
  });
  return fn;
}

// Byte tensor of rank 4, innermost dimension contiguous; box = {box0, box1, box2, box3} bytes /
// rows; 64-byte swizzle when the innermost box is 64 bytes.
// bf16 output tensor (B, Sq, Hq, Dv) as {Dv, Hq, Sq, B}; box = 64 columns x `rows` rows, 128-byte
// swizzle (the staging layout of the warp-specialised kernels' epilogues).
bool encode_out_4d(CUtensorMap* m, void* base, const uint64_t (&dims)[4], const uint64_t (&strides)[3], uint32_t rows) {
  auto fn = get_encode();
  if (fn == nullptr) return false;
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  const cuuint32_t box[4] = {64, 1, rows, 1};
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, base, dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

bool encode_u8_4d(CUtensorMap* m, const void* base, const uint64_t (&dims)[4],
                  const uint64_t (&strides)[3], const uint32_t (&box)[4], CUtensorMapSwizzle sw) {
  auto fn = get_encode();
  if (fn == nullptr) return false;
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<void*>(base), dims, strides,
                        box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// Launch epoch recorded with a device-side failure (see ptx.cuh): launches modulo 256.
uint32_t next_launch_epoch() {
  static std::atomic<uint32_t> counter{0};
  return counter.fetch_add(1, std::memory_order_relaxed) & 0xffu;
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Per-kernel launch preparation, done once per (kernel, device) and remembered: the opt-in to
// `smem_bytes` of dynamic shared memory, the carve-out (see launch_pdl) and -- for the warp-specialised kernels, which re-partition
// registers with setmaxnreg -- the check that the build kept the register count the budget in the
// source assumes (an increase blocks for ever when the CTA was launched with fewer registers per
// thread; such a build is refused with -FA4_E_BUILD instead of being launched).
// expected_regs = 0: no register check.
int prepare_kernel(const void* kernel, uint32_t smem_bytes, int expected_regs) {
  static std::mutex mu;
  static std::map<std::pair<const void*, int>, int> seen;   // -> result of the first preparation
  int dev = 0;
  const cudaError_t ge = cudaGetDevice(&dev);
  if (ge != cudaSuccess) return (int)ge;
  std::lock_guard<std::mutex> lock(mu);
  const auto key = std::make_pair(kernel, dev);
  const auto it = seen.find(key);
  if (it != seen.end()) return it->second;
  int rc = 0;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return (int)e;          // not remembered: the caller may retry
  if (expected_regs > 0) {
    cudaFuncAttributes attr;
    e = cudaFuncGetAttributes(&attr, kernel);
    if (e != cudaSuccess) return (int)e;
    if (attr.numRegs < expected_regs) rc = -FA4_E_BUILD;
  }
  seen[key] = rc;
  return rc;
}
template <class Kernel>
int ensure_smem(Kernel kernel, uint32_t bytes) {
  return prepare_kernel(reinterpret_cast<const void*>(kernel), bytes, 0);
}
template <class Kernel>
int ensure_kernel(Kernel kernel, uint32_t bytes, int expected_regs) {
  return prepare_kernel(reinterpret_cast<const void*>(kernel), bytes, expected_regs);
}

// Launch as a programmatic dependent of whatever precedes it in the stream (see pdl_wait in
// ptx.cuh): launch latency and set-up overlap the end of the kernel before.
// Every kernel asks for the largest shared-memory carve-out, also those that use none: an SM changes
// its carve-out only while it is empty, which would take the overlap away again.
template <class... KArgs, class... Args>
int launch_pdl_cluster(unsigned cluster, void (*kernel)(KArgs...), dim3 grid, unsigned threads, uint32_t smem,
                       cudaStream_t stream, Args&&... args) {
  if (int e = prepare_kernel(reinterpret_cast<const void*>(kernel), smem, 0)) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim = {cluster, 1, 1};
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return (int)cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
template <class Kernel, class... Args>
int launch_pdl(Kernel kernel, dim3 grid, unsigned threads, uint32_t smem, cudaStream_t stream, Args&&... args) {
  return launch_pdl_cluster(1, kernel, grid, threads, smem, stream, std::forward<Args>(args)...);
}

// How many clusters of `cluster` CTAs can be resident at once (asked once per kernel, size and device;
// 0 if the runtime cannot say).
int clusters_at_once(const void* kernel, int cluster, unsigned threads, uint32_t smem) {
  static std::mutex mu;
  static std::map<std::pair<const void*, std::pair<int, int>>, int> seen;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> lock(mu);
  const auto key = std::make_pair(kernel, std::make_pair(cluster, dev));
  const auto it = seen.find(key);
  if (it != seen.end()) return it->second;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)cluster);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim = {(unsigned)cluster, 1, 1};
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    n = 0;
  }
  return seen[key] = n;
}

}  // namespace

extern "C" int fa4_nvfp4_query(int32_t what) {
  static const int dims[] = {128, 64, 192};   // 192 pairs with a V / O head dim of 128
  switch (what) {
    case 0: return FA4_NVFP4_ABI_VERSION;
    case 1: return (int)(sizeof(dims) / sizeof(dims[0]));
    case 100: return (int)fa4::ws::kSmemRequest;
    case 101: return (int)fa4::kEx2EmuMask;
    case 102: return FA4_P_SCALE_E4M3;
    default:
      if (what >= 2 && what < 2 + (int)(sizeof(dims) / sizeof(dims[0]))) return dims[what - 2];
      return -FA4_E_SHAPE;
  }
}

namespace {
// Whether the decode kernel merges the splits of an entry itself, as one cluster: up to eight (the
// portable cluster size), while all CTAs are resident at once.  Beyond that the clusters start unevenly
// (B=64, Sk=4096, two splits, 1024 CTAs: 64 us with the combine kernel, 68 with clusters; one token at
// Sk=777, 24 CTAs: 8.8 and 7.7).  A single split needs neither.
bool decode_in_cluster(const fa4_nvfp4_params* p, int num_splits) {
  const int64_t ctas = (int64_t)num_splits * p->Hkv * p->B;
  const int64_t resident = kSms * (p->Sq * (p->Hq / p->Hkv) <= 16 ? 3 : 2);
  return num_splits == 1 || (num_splits <= dec::kMaxCluster && ctas <= resident);
}
// The balanced form of a decode call (entries of unequal lengths, see balance() in attn_decode.cuh).
constexpr int kSortedUnits = 200;       // units from which on entries come by length
int balanced_slots(const fa4_nvfp4_params* p) { return (int)kSms * (p->Sq * (p->Hq / p->Hkv) <= 16 ? 3 : 2); }
// One CTA a place and piece; or, with (nearly) as many units as places, what the units need and a quarter more to cut the
// long ones.  (Half and a tenth as many more: 64 entries up to 8192 keys, 8 heads 41.3, 39.9 us, with a quarter 38.6.)
int balanced_ctas(const fa4_nvfp4_params* p) {
  const int units = p->B * p->Hkv, slots = balanced_slots(p);
  return units + slots / 16 <= slots ? slots : units + slots / 4;
}
int64_t balanced_bytes(const fa4_nvfp4_params* p) {
  // partial O and LSE of a CTA, then the table of pieces
  const int64_t rows = (int64_t)balanced_ctas(p) * p->Sq * (p->Hq / p->Hkv);
  return rows * 129 * 4 + 16 + (int64_t)p->B * p->Hkv * 8;
}
// Whether a decode call with key counts in memory is dealt by the lengths.  The host knows the longest possible length
// alone.  Dealing costs 3 us (1.3 in front of the first load, the rest the second launch, of which 1.2 where nothing is merged), so it takes that many blocks
// (times kv heads, over the batch) for the unevenness to cost more.  us, splits of equal number / dealt, lengths
// spread over the logarithm down to a 64th of the longest, GQA 4:
//   one token, 2048 blocks: 5, 8, 16, 32 entries of 8 heads 9.5 / 10.6, 9.9 / 10.6, 8.8 / 9.3, 8.9 / 11.3; 4096: 14.4 / 14.5, 15.2 /
//     14.8, 11.5 / 10.5, 11.2 / 11.7, 3 entries 17.1 / 18.9; 8192: 25.1 / 23.1, 21.0 / 16.6, 18.5 / 14.6, 20.0 / 15.8, 3
//     entries 21.6 / 21.1, 48 entries 19.7 / 18.8, 64 entries (more units than places) 21.9 / 22.9; 16384: 38.7 / 34.6,
//     39.9 / 30.3, 34.8 / 26.9, 33.8 / 23.3; 3, 48, 64 entries 36.4 / 33.0, 31.7 / 24.4, 29.6 / 30.3; 32768: 64 entries
//     41.2 / 38.6; two entries never gain (16384: 43.1 / 43.4)
//   32 heads, 8 entries, 4096, 8192, 32768 blocks 13.0 / 13.8, 20.8 / 17.3, 58.6 / 33.5; 24 entries 13.7 / 17.6, 17.5 / 21.8,
//     38.5 / 36.5; 40 entries, 32768, 81920 41.2 / 49.8, 81 / 81
//   four tokens (16 rows), 1024 blocks: 6, 16 entries 9.9 / 11.0, 9.7 / 10.9; 2048: 13.8 / 12.3, 12.4 / 10.5; 4096: 21.8 / 18.1,
//     19.2 / 12.5; eight (32 rows): 1024: 16.4 / 13.6, 13.3 / 13.9; 2048: 18.3 / 16.2, 16.7 / 12.5; 4096: 30.4 / 23.8, 26.7 / 16.4
// (Above eight rows a block takes one softmax warpgroup longer, so a long entry costs more.)
// A batch of few units is cut into the more pieces each (444 places), and the second launch merges them row by
// row: the line rises as the units become fewer.  us, equal / dealt, one kv head unless two are given, last equal and first
// faster one:
//   8 rows: 5 units 20000 blocks 43.5 / 47.5, 32000 71.3 / 67.5; 8: 13000 31.3 / 33.2, 20000 40.8 / 38.1; 16: 6500 20.0 /
//     20.6, 9000 23.0 / 21.5; 32: 6500 19.7 / 17.6; 4 rows, two heads, 10: 13000 30.5 / 30.9, 20000 45.6 / 41.3
//   16 rows: 3: 16000 62.4 / 66.9, 24000 77.7 / 64.1; 4: 2200 14.2 / 23.5, 12000 49.0 / 49.5, 16000 57.5 / 49.0; 8: 6500 25.5 /
//     26.7, 9000 36.2 / 30.4; 16, two heads: 3200 17.1 / 17.7, 4500 21.3 / 20.2; 20: 3300 16.1 /
//     16.8; 32: 2200 14.0 / 12.4
//   32 rows: 4: 6500 42.9 / 45.6, 9000 46.4 / 41.7; 8: 2200 19.2 / 19.5, 3200 24.8 / 23.1; 16: 2200 17.5 / 15.4
// All of these are lengths spread over the logarithm.  Where the lengths do not differ, or are all short, dealing gains nothing, and
// the call is slower by what it costs; the host cannot tell.  us, equal splits / dealt, GQA 4, 8 kv heads, one token, tiled scales; all
// entries full, between half and full, uniform, spread as above, one full and the others a 32nd, all a tenth, all 300 keys:
//   16 x 4096: 18.8 / 21.4, 17.0 / 19.4, 14.9 / 15.1, 11.2 / 10.5, 10.7 / 9.8, 7.4 / 8.7, 7.3 / 8.2
//   8 x 8192: 18.5 / 21.6, 17.3 / 19.2, 16.3 / 18.1, 15.1 / 14.9, 12.8 / 10.8, 7.3 / 9.6, 6.7 / 8.0
//   16 x 8192: 32.0 / 35.1, 26.1 / 28.5, 21.4 / 20.1, 16.7 / 13.8, 15.8 / 10.9, 8.1 / 11.5, 7.3 / 8.1
//   32 x 8192: 55.4 / 55.2, 46.6 / 51.7, 37.8 / 37.9, 33.5 / 20.7, 25.5 / 12.9, 8.8 / 11.4, 6.7 / 8.8
//   64 x 8192 (more units than places): 108 / 135, 90.4 / 96.8, 68.1 / 68.5, 42.6 / 38.9, 25.6 / 22.1, 31.8 / 21.1, 26.1 / 15.0
//   16 x 32768: 107 / 113, 78.5 / 79.4, 56.1 / 45.3, 63.9 / 40.2, 46.3 / 18.2, 13.0 / 17.6, 7.3 / 8.2
//   four tokens, 8 x 4096: 16.5 / 20.0, 14.8 / 17.5, 13.4 / 15.3, 12.3 / 11.9, 11.2 / 11.1, 7.3 / 9.1, 7.3 / 9.3
//   16 x 8192: 39.7 / 43.0, 38.0 / 33.7, 36.9 / 25.4, 32.7 / 16.6, 31.6 / 12.8, 9.5 / 13.9, 7.7 / 9.5
//   linear scales, which equal splits have tiled first, 8 x 8192: 24.4 / 30.1, 23.7 / 25.8, 22.1 / 23.5, 21.3 / 19.6, 17.1 / 13.8, 13.6 /
//     12.6, 12.9 / 10.1; 16 x 8192: 43.9 / 47.9, 37.6 / 38.9, 32.4 / 28.5, 28.2 / 18.4, 27.0 / 13.8, 19.0 / 15.2, 17.6 / 10.2
// Over the seven and lengths spread down to an eighth, dealing is even in the mean at 8192 blocks (4096 above eight rows), gains up to
// 39 % beyond (linear scales 56), and at half of that loses 5 to 14 % with tiled scales and gains 3 to 27 % with linear ones: the
// line stays between the two.  A caller who knows that lengths are even gives a split count, see dealt_bytes().
bool decode_balanced(const fa4_nvfp4_params* p, const int32_t* seqused_k) {
  if (seqused_k == nullptr || p->B < 3 || p->B > dec::kMaxBalanced || p->Sk > dec::kMaxBalancedKeys) return false;
  const int64_t units = (int64_t)p->B * p->Hkv, blocks = units * ((p->Sk + kBlockN - 1) / kBlockN);
  const int slots = balanced_slots(p);
  if (units > 2 * slots || balanced_ctas(p) > dec::kMaxBalancedCtas || blocks > dec::kMaxBalancedBlocks) return false;
  if (units > slots) return blocks >= 40 * units;
  const int rows = p->Sq * (p->Hq / p->Hkv);
  const int64_t least = rows > 8 ? 2048 : (units < 40 ? 6144 : 4096);
  const int64_t few = units >= 32 ? 0 : (rows > 16 ? 32000 : (rows > 8 ? 72000 : 144000)) / units;
  return blocks >= std::max({least, few, 24 * units});
}
int64_t splitkv_bytes(const fa4_nvfp4_params* p, int num_splits) {
  // partial O (num_splits, B, Sq, Hq, Dv) fp32, then partial LSE (num_splits, B, Hq, Sq) fp32
  return (int64_t)num_splits * p->B * p->Sq * p->Hq * ((int64_t)p->Dv + 1) * 4;
}
// Workspace with which a call is dealt by the lengths: more than its splits need, so that a caller who has room for those alone
// gets them, whatever their number.
int64_t dealt_bytes(const fa4_nvfp4_params* p, int num_splits) {
  return (decode_in_cluster(p, num_splits) ? 0 : splitkv_bytes(p, num_splits)) + balanced_bytes(p);
}
// KV-cache view of K / V: per-entry key counts and / or a page pool (see fa4_nvfp4_ext).
struct CacheView {
  const int32_t* seqused_k = nullptr;
  const int32_t* page_table = nullptr;
  int page_size = 0, pages_per_seq = 0, num_pages = 0;
  // packed variable-length batch (see fa4_nvfp4_varlen)
  const int32_t* cu_seqlens_q = nullptr;
  const int32_t* cu_seqlens_k = nullptr;
  const int32_t* cu_seqlens_v = nullptr;   // starts inside V (multiples of 32); null: cu_seqlens_k
  int total_q = 0, total_k = 0, total_v = 0;
};
int launch_fwd(const fa4_nvfp4_params* p, int num_splits, void* workspace, uint64_t workspace_bytes,
               int win_left, int win_right, const float* sink, float softcap, const CacheView& cache,
               void* cuda_stream, const float* const* scales = nullptr, const fa4_nvfp4_linear_sf* linear = nullptr);
}  // namespace

extern "C" int fa4_nvfp4_fwd(const fa4_nvfp4_params* p, void* cuda_stream) {
  return launch_fwd(p, 1, nullptr, 0, -1, -1, nullptr, 0.f, CacheView{}, cuda_stream);
}

namespace {
int fwd_ex(const fa4_nvfp4_params* p, const fa4_nvfp4_ext* x, const float* const* scales, void* cuda_stream,
           const fa4_nvfp4_linear_sf* linear = nullptr) {
  if (x == nullptr) return -FA4_E_NULL;
  if (x->struct_size != sizeof(fa4_nvfp4_ext)) return -FA4_E_STRUCT;
  const int splits = x->num_splits == 0 ? 1 : x->num_splits;
  if (splits < 1 || splits > 128 || x->window_left < -1 || x->window_right < -1) return -FA4_E_SHAPE;
  if (!(x->softcap >= 0.f) || x->softcap > 3.0e38f || x->reserved != 0u) return -FA4_E_SHAPE;
  CacheView cache;
  cache.seqused_k = x->seqused_k;
  if (x->page_table != nullptr) {
    // pages hold whole 128-key blocks; the table must cover the logical key length
    if (x->page_size <= 0 || x->page_size % 128 != 0 || x->num_pages <= 0 || x->pages_per_seq <= 0)
      return -FA4_E_SHAPE;
    if (p != nullptr && (int64_t)x->pages_per_seq * x->page_size < p->Sk) return -FA4_E_SHAPE;
    cache.page_table = x->page_table;
    cache.page_size = x->page_size;
    cache.pages_per_seq = x->pages_per_seq;
    cache.num_pages = x->num_pages;
  }
  return launch_fwd(p, splits, x->workspace, x->workspace_bytes, x->window_left, x->window_right,
                    x->sink, x->softcap, cache, cuda_stream, scales, linear);
}
}  // namespace

extern "C" int fa4_nvfp4_fwd_ex(const fa4_nvfp4_params* p, const fa4_nvfp4_ext* x, void* cuda_stream) {
  return fwd_ex(p, x, nullptr, cuda_stream);
}

extern "C" int fa4_nvfp4_fwd_device_scales(const fa4_nvfp4_params* p, const fa4_nvfp4_ext* x, const float* q_scale,
                                           const float* k_scale, const float* v_scale, void* cuda_stream) {
  if (p == nullptr || !q_scale || !k_scale || !v_scale) return -FA4_E_NULL;
  fa4_nvfp4_params q = *p;
  q.q_scale = q.k_scale = q.v_scale = 1.f;      // not read
  const float* const scales[3] = {q_scale, k_scale, v_scale};
  return fwd_ex(&q, x, scales, cuda_stream);
}

extern "C" int fa4_nvfp4_fwd_decode_linear_sf(const fa4_nvfp4_params* p, const fa4_nvfp4_ext* x,
                                              const fa4_nvfp4_linear_sf* sf, void* cuda_stream) {
  if (p == nullptr || sf == nullptr) return -FA4_E_NULL;
  if (sf->struct_size != sizeof(fa4_nvfp4_linear_sf) || sf->reserved != 0u) return -FA4_E_STRUCT;
  if (p->variant != FA4_VARIANT_DECODE) return -FA4_E_VARIANT;
  // the producers walk upwards from the pointers they are given, as for the data; 0 repeats a row
  const int64_t strides[] = {sf->q_stride_b, sf->q_stride_s, sf->q_stride_h, sf->k_stride_b, sf->k_stride_s,
                             sf->k_stride_h, sf->v_stride_b, sf->v_stride_h, sf->v_stride_d};
  for (int64_t s : strides)
    if (s < 0) return -FA4_E_STRIDE;
  if (sf->q_scale == nullptr && sf->k_scale == nullptr && sf->v_scale == nullptr)
    return fwd_ex(p, x, nullptr, cuda_stream, sf);
  if (!sf->q_scale || !sf->k_scale || !sf->v_scale) return -FA4_E_NULL;
  fa4_nvfp4_params q = *p;
  q.q_scale = q.k_scale = q.v_scale = 1.f;      // not read
  const float* const scales[3] = {sf->q_scale, sf->k_scale, sf->v_scale};
  return fwd_ex(&q, x, scales, cuda_stream, sf);
}

extern "C" int fa4_nvfp4_fwd_varlen(const fa4_nvfp4_params* p, const fa4_nvfp4_varlen* v, void* cuda_stream) {
  if (p == nullptr || v == nullptr) return -FA4_E_NULL;
  if (v->struct_size != sizeof(fa4_nvfp4_varlen) || p->struct_size != sizeof(fa4_nvfp4_params)) return -FA4_E_STRUCT;
  if (v->cu_seqlens_q == nullptr || v->cu_seqlens_k == nullptr) return -FA4_E_NULL;
  if (v->num_seqs <= 0 || v->total_q <= 0 || v->total_k <= 0 || v->max_seqlen_q <= 0 || v->max_seqlen_k <= 0 ||
      v->max_seqlen_q > v->total_q || v->max_seqlen_k > v->total_k)
    return -FA4_E_SHAPE;
  if (v->window_left < -1 || v->window_right < -1 || !(v->softcap >= 0.f) || v->softcap > 3.0e38f || v->reserved != 0u ||
      v->reserved2 != 0)
    return -FA4_E_SHAPE;
  if (v->cu_seqlens_v != nullptr ? (v->total_v < v->total_k || v->total_v % 32 != 0) : v->total_v != 0)
    return -FA4_E_SHAPE;
  if (p->variant != FA4_VARIANT_AUTO && p->variant != FA4_VARIANT_WS64) return -FA4_E_VARIANT;
  // one launch over (sequence, m-block of the longest sequence, head): the grid of the dense call
  // with B = number of sequences and Sq / Sk = the longest ones
  fa4_nvfp4_params q = *p;
  q.B = v->num_seqs;
  q.Sq = v->max_seqlen_q;
  q.Sk = v->max_seqlen_k;
  q.variant = FA4_VARIANT_WS64;
  CacheView cache;
  cache.seqused_k = v->seqused_k;
  cache.cu_seqlens_q = v->cu_seqlens_q;
  cache.cu_seqlens_k = v->cu_seqlens_k;
  cache.total_q = v->total_q;
  cache.total_k = v->total_k;
  cache.cu_seqlens_v = v->cu_seqlens_v;
  cache.total_v = v->cu_seqlens_v != nullptr ? v->total_v : v->total_k;
  return launch_fwd(&q, 1, nullptr, 0, v->window_left, v->window_right, v->sink, v->softcap, cache, cuda_stream);
}

extern "C" int fa4_nvfp4_sf_tile_jobs(const fa4_nvfp4_sf_job* jobs, int32_t n, void* cuda_stream) {
  if (jobs == nullptr) return -FA4_E_NULL;
  if (n < 1 || n > 3) return -FA4_E_SHAPE;
  SfTileJobs k;
  k.n = n;
  int64_t blocks = 0;
  for (int i = 0; i < n; ++i) {
    const fa4_nvfp4_sf_job& a = jobs[i];
    SfTileJob& j = k.job[i];
    if (!a.src || !a.dst) return -FA4_E_NULL;
    if (a.n_outer <= 0 || a.n_inner <= 0 || a.rows <= 0 || a.cols <= 0 || a.col_tile_multiple <= 0) return -FA4_E_SHAPE;
    if (!aligned16(a.dst)) return -FA4_E_ALIGN;
    j.src = static_cast<const uint8_t*>(a.src);
    j.dst = static_cast<uint8_t*>(a.dst);
    j.cu = a.cu_seqlens;
    j.packed_rows = a.packed_rows ? 1 : 0;
    j.stride_outer = a.stride_outer;
    j.stride_inner = a.stride_inner;
    j.stride_row = a.stride_row;
    j.n_inner = a.n_inner;
    j.rows = a.rows;
    j.cols = a.cols;
    j.row_tiles = (a.rows + 127) / 128;
    j.col_tiles = ((a.cols + 3) / 4 + a.col_tile_multiple - 1) / a.col_tile_multiple * a.col_tile_multiple;
    const int64_t combos = (int64_t)a.n_inner * j.col_tiles;
    const int64_t warps = (int64_t)a.n_outer * j.row_tiles * ((combos + 7) / 8) * 8;
    if (combos > 0x7fffffffll || warps > 0x7fffffffll) return -FA4_E_TOO_LARGE;
    j.combos = (int)combos;
    j.warps = (uint32_t)warps;
    j.first_block = (int)blocks;
    j.div_combo8 = make_fastdiv((uint32_t)((combos + 7) / 8));
    j.div_row_tiles = make_fastdiv((uint32_t)j.row_tiles);
    j.div_col_tiles = make_fastdiv((uint32_t)j.col_tiles);
    blocks += (warps + 7) / 8;
  }
  if (blocks > 0x7fffffffll) return -FA4_E_TOO_LARGE;
  return launch_pdl(sf_tile_kernel, dim3((unsigned)blocks), 256, 0, static_cast<cudaStream_t>(cuda_stream), k);
}

extern "C" int fa4_nvfp4_sf_linear_to_tiled_packed(const void* src, void* dst, const int32_t* cu_seqlens,
                                                   int32_t num_seqs, int32_t n_inner, int32_t max_rows,
                                                   int32_t max_cols, int64_t stride_inner, int64_t stride_row,
                                                   int32_t col_tile_multiple, int32_t packed_rows,
                                                   void* cuda_stream) {
  if (!cu_seqlens) return -FA4_E_NULL;
  const fa4_nvfp4_sf_job j = {src, dst, cu_seqlens, num_seqs, n_inner, max_rows, max_cols, 0, stride_inner, stride_row,
                              col_tile_multiple, packed_rows};
  return fa4_nvfp4_sf_tile_jobs(&j, 1, cuda_stream);
}

extern "C" int64_t fa4_nvfp4_splitkv_workspace_bytes(const fa4_nvfp4_params* p, int32_t num_splits) {
  if (p == nullptr || p->struct_size != sizeof(fa4_nvfp4_params)) return -FA4_E_STRUCT;
  if (num_splits < 1 || num_splits > 128 || p->B <= 0 || p->Sq <= 0 || p->Hq <= 0 || p->Dv <= 0)
    return -FA4_E_SHAPE;
  if (p->variant == FA4_VARIANT_DECODE && p->Hkv > 0 && p->Hq >= p->Hkv && decode_in_cluster(p, num_splits)) return 0;
  return num_splits == 1 ? 0 : splitkv_bytes(p, num_splits);
}

extern "C" int fa4_nvfp4_decode_is_balanced(int32_t B, int32_t Sq, int32_t Sk, int32_t Hq, int32_t Hkv) {
  fa4_nvfp4_params p = {};
  p.B = B; p.Sq = Sq; p.Sk = Sk; p.Hq = Hq; p.Hkv = Hkv;
  const int32_t any = 0;      // (only whether there are counts matters)
  return B > 0 && Sq > 0 && Sk > 0 && Hkv > 0 && Hq >= Hkv && decode_balanced(&p, &any) ? 1 : 0;
}

extern "C" int64_t fa4_nvfp4_fwd_ex_workspace_bytes(const fa4_nvfp4_params* p, const fa4_nvfp4_ext* x) {
  if (x == nullptr) return -FA4_E_NULL;
  if (x->struct_size != sizeof(fa4_nvfp4_ext)) return -FA4_E_STRUCT;
  const int64_t bytes = fa4_nvfp4_splitkv_workspace_bytes(p, x->num_splits == 0 ? 1 : x->num_splits);
  if (bytes < 0 || p->variant != FA4_VARIANT_DECODE || p->Hkv <= 0 || p->Hq < p->Hkv || !decode_balanced(p, x->seqused_k))
    return bytes;
  return dealt_bytes(p, x->num_splits == 0 ? 1 : x->num_splits);
}

extern "C" int fa4_nvfp4_fwd_splitkv(const fa4_nvfp4_params* p, int32_t num_splits, void* workspace,
                                     uint64_t workspace_bytes, void* cuda_stream) {
  if (num_splits < 1 || num_splits > 128) return -FA4_E_SHAPE;
  return launch_fwd(p, num_splits, workspace, workspace_bytes, -1, -1, nullptr, 0.f, CacheView{}, cuda_stream);
}

namespace {
// What a call resolves to once its arguments have been accepted.
struct FwdPlan {
  int variant = 0;
  int win_left = -1, win_right = -1;
  bool decode = false, balanced = false, d192 = false, local = false, general = false, cached = false;
  int dec_rows = 0;
};

// Every host-side check of a forward call.  Touches no CUDA API: a call that fails here has
// launched nothing and has not made a device current.  `linear_sf`: the three scale pointers are
// the caller's LINEAR layouts (the allocation-free entry point), which need no 16-byte alignment.
int validate_fwd(const fa4_nvfp4_params* p, int num_splits, const void* workspace, uint64_t workspace_bytes,
                 int win_left, int win_right, const float* sink, float softcap, const CacheView& cache,
                 bool linear_sf, FwdPlan* plan) {
  if (p == nullptr) return -FA4_E_NULL;
  if (p->struct_size != sizeof(fa4_nvfp4_params)) return -FA4_E_STRUCT;
  if (!p->q || !p->k || !p->v || !p->q_sf || !p->k_sf || !p->v_sf || !p->out) return -FA4_E_NULL;
  if (p->B <= 0 || p->Sq <= 0 || p->Sk <= 0 || p->Hq <= 0 || p->Hkv <= 0) return -FA4_E_SHAPE;
  if (p->Hq % p->Hkv != 0) return -FA4_E_SHAPE;
  // head dims built: (128, 128), (64, 64) and (192, 128), the last on the 64-key kernel only
  const bool d192 = p->D == 192 && p->Dv == 128;
  if (!d192 && (p->D != p->Dv || (p->D != 128 && p->D != 64))) return -FA4_E_SHAPE;
  // Sq and Sk are free.  V is stored key-contiguous with its key axis padded to a multiple of 32
  // (zero values, zero scales): keys are blocked by 16 along that axis and the 16-byte stride rule
  // of TMA (checked below) needs whole 32-key groups per row; keys >= Sk are masked
  if ((int64_t)((p->Sq + kBlockM - 1) / kBlockM) * p->Hq * p->B > 0x7fffffffLL) return -FA4_E_SHAPE;
  if (!(p->softmax_scale > 0.f) || !(p->q_scale > 0.f) || !(p->k_scale > 0.f)) return -FA4_E_SHAPE;
  const void* ptrs[] = {p->q, p->k, p->v, p->out};
  for (const void* q : ptrs)
    if (!aligned16(q)) return -FA4_E_ALIGN;
  if (!linear_sf && (!aligned16(p->q_sf) || !aligned16(p->k_sf) || !aligned16(p->v_sf))) return -FA4_E_ALIGN;
  const int64_t bstr[] = {p->q_stride_b, p->q_stride_s, p->q_stride_h, p->k_stride_b, p->k_stride_s,
                          p->k_stride_h, p->v_stride_b, p->v_stride_h, p->v_stride_d};
  for (int64_t s : bstr)
    if (s <= 0 || (s & 15) != 0) return -FA4_E_STRIDE;
  if ((p->o_stride_b & 7) || (p->o_stride_s & 7) || (p->o_stride_h & 7)) return -FA4_E_STRIDE;
  // automatic choice: the 64-key kernel where it applies (no split-KV), the 128-key kernel
  // otherwise
  const bool cached = cache.seqused_k != nullptr || cache.page_table != nullptr || cache.cu_seqlens_q != nullptr;
  const bool takes64 = num_splits == 1;   // what the 64-key kernel can run
  int variant = p->variant;
  if (variant == FA4_VARIANT_AUTO) variant = takes64 ? FA4_VARIANT_WS64 : FA4_VARIANT_WS;
  if (variant != FA4_VARIANT_WS && variant != FA4_VARIANT_WS64 && variant != FA4_VARIANT_DECODE)
    return -FA4_E_VARIANT;
  const bool decode = variant == FA4_VARIANT_DECODE;
  if (decode) {
    // a handful of query rows per kv head, head dim 128, causal or unmasked
    if (p->D != 128 || p->Dv != 128 || (int64_t)p->Sq * (p->Hq / p->Hkv) > dec::kMaxRows) return -FA4_E_SHAPE;
    if (win_left >= 0 || win_right > 0 || sink != nullptr || softcap > 0.f) return -FA4_E_SHAPE;
    plan->balanced = workspace != nullptr && aligned16(workspace) && decode_balanced(p, cache.seqused_k) &&
                     workspace_bytes >= (uint64_t)dealt_bytes(p, num_splits);
    if (!plan->balanced && !decode_in_cluster(p, num_splits)) {
      if (workspace == nullptr || !aligned16(workspace)) return -FA4_E_NULL;
      if (workspace_bytes < (uint64_t)splitkv_bytes(p, num_splits)) return -FA4_E_TOO_LARGE;
    }
  }
  if (variant == FA4_VARIANT_WS64 && !takes64) return -FA4_E_SHAPE;
  if (d192 && variant != FA4_VARIANT_WS64) return -FA4_E_SHAPE;
  // window limits: `causal` is the right limit 0; an explicit right limit overrides it
  if (p->causal && win_right < 0) win_right = 0;
  const bool local = win_left >= 0 || win_right > 0;
  if (num_splits > 1 && !decode) {
    if (workspace == nullptr) return -FA4_E_NULL;
    if (!aligned16(workspace)) return -FA4_E_ALIGN;
    if (workspace_bytes < (uint64_t)splitkv_bytes(p, num_splits)) return -FA4_E_TOO_LARGE;
    if ((int64_t)((p->Sq + kBlockM - 1) / kBlockM) * p->Hq * p->B * num_splits > 0x7fffffffLL)
      return -FA4_E_SHAPE;
  }
  plan->variant = variant;
  plan->win_left = win_left;
  plan->win_right = win_right;
  plan->decode = decode;
  plan->d192 = d192;
  plan->local = local;
  plan->cached = cached;
  plan->general = local || num_splits > 1 || sink != nullptr || softcap > 0.f || cached;
  plan->dec_rows = p->Sq * (p->Hq / p->Hkv);
  return 0;
}

int launch_fwd(const fa4_nvfp4_params* p, int num_splits, void* workspace, uint64_t workspace_bytes,
               int win_left, int win_right, const float* sink, float softcap, const CacheView& cache,
               void* cuda_stream, const float* const* scales, const fa4_nvfp4_linear_sf* linear) {
  FwdPlan plan;
  if (int e = validate_fwd(p, num_splits, workspace, workspace_bytes, win_left, win_right, sink, softcap, cache,
                           linear != nullptr, &plan))
    return e;
  const int variant = plan.variant;
  const bool decode = plan.decode, local = plan.local, general = plan.general, cached = plan.cached;
  const int dec_rows = plan.dec_rows;
  win_left = plan.win_left;
  win_right = plan.win_right;

  CUtensorMap tm_q, tm_k, tm_v;
  {
    // a packed batch is one long sequence for the tensor maps: the kernel adds each sequence's
    // first row to the row coordinate
    const bool packed = cache.cu_seqlens_q != nullptr;
    const uint64_t dq[4] = {(uint64_t)p->D / 2, (uint64_t)p->Hq, packed ? (uint64_t)cache.total_q : (uint64_t)p->Sq,
                            packed ? 1u : (uint64_t)p->B};
    const uint64_t sq[3] = {(uint64_t)p->q_stride_h, (uint64_t)p->q_stride_s, (uint64_t)p->q_stride_b};
    // a Q / K tile row is D / 2 bytes: one 64-byte-swizzled box for D = 128; 32-byte-wide boxes
    // (32-byte swizzle), one per 64-element step, for D = 64 and 192
    const uint32_t qk_box = p->D == 128 ? 64u : 32u;
    const uint32_t bq[4] = {qk_box, 1, (uint32_t)kBlockM, 1};
    // with a page table K / V describe the pool: "batch" = page, "Sk" = keys per page
    const uint64_t k_rows = cache.page_table ? (uint64_t)cache.page_size
                                             : (packed ? (uint64_t)cache.total_k : (uint64_t)p->Sk);
    const uint64_t k_batch = cache.page_table ? (uint64_t)cache.num_pages : (packed ? 1u : (uint64_t)p->B);
    const uint64_t dk[4] = {(uint64_t)p->D / 2, (uint64_t)p->Hkv, k_rows, k_batch};
    const uint64_t sk[3] = {(uint64_t)p->k_stride_h, (uint64_t)p->k_stride_s, (uint64_t)p->k_stride_b};
    const uint32_t bk[4] = {qk_box, 1, (uint32_t)kBlockN, 1};
    const uint64_t v_keys = packed ? (uint64_t)cache.total_v : k_rows;   // a packed V has its own, padded key axis
    const uint64_t dv[4] = {(v_keys + 31) / 32 * 16, (uint64_t)p->Dv, (uint64_t)p->Hkv, k_batch};   // padded key axis
    const uint64_t sv[3] = {(uint64_t)p->v_stride_d, (uint64_t)p->v_stride_h, (uint64_t)p->v_stride_b};
    const uint32_t bv[4] = {64, (uint32_t)p->Dv, 1, 1};
    // a Q / K tile row is D / 2 bytes: 64-byte swizzle for D = 128, 32-byte for D = 64
    const CUtensorMapSwizzle sw_qk = p->D == 128 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
    if (!encode_u8_4d(&tm_q, p->q, dq, sq, bq, sw_qk) ||
        !encode_u8_4d(&tm_k, p->k, dk, sk, bk, sw_qk) ||
        !encode_u8_4d(&tm_v, p->v, dv, sv, bv, CU_TENSOR_MAP_SWIZZLE_64B))
      return -FA4_E_TENSORMAP;
  }

  KernelParams kp;
  kp.q_sf = static_cast<const uint8_t*>(p->q_sf);
  kp.k_sf = static_cast<const uint8_t*>(p->k_sf);
  kp.v_sf = static_cast<const uint8_t*>(p->v_sf);
  kp.out = static_cast<__nv_bfloat16*>(p->out);
  kp.lse = p->lse;
  kp.status = p->status;
  kp.epoch = next_launch_epoch();
  kp.o_stride_b = p->o_stride_b;
  kp.o_stride_s = p->o_stride_s;
  kp.o_stride_h = p->o_stride_h;
  kp.B = p->B; kp.Sq = p->Sq; kp.Sk = p->Sk; kp.Hq = p->Hq; kp.Hkv = p->Hkv;
  kp.group = p->Hq / p->Hkv;
  kp.div_tiles_per_m = make_fastdiv((uint32_t)p->Hq * (uint32_t)p->B);
  kp.div_hq = make_fastdiv((uint32_t)p->Hq);
  kp.div_group = make_fastdiv((uint32_t)kp.group);
  kp.div_splits = make_fastdiv((uint32_t)num_splits);
  kp.div_page = make_fastdiv(cache.page_table != nullptr ? (uint32_t)(cache.page_size / kBlockN) : 1u);
  kp.num_m_blocks = (p->Sq + kBlockM - 1) / kBlockM;
  kp.num_n_blocks = (p->Sk + kBlockN - 1) / kBlockN;
  kp.causal = win_right >= 0 ? 1 : 0;
  kp.win_left = win_left;
  kp.win_right = win_right;
  kp.sink = sink;
  // tiled scale factors: (B, H, row tiles, col tiles, 512)
  kp.qsf_stride_h = (int64_t)kp.num_m_blocks * (p->D / 64) * 512;
  kp.qsf_stride_b = kp.qsf_stride_h * p->Hq;
  // (per page when K / V are a page pool: the tiled scales of a page are laid out like those of
  // a batch entry of page_size keys)
  const int64_t kv_blocks = cache.page_table ? cache.page_size / kBlockN : kp.num_n_blocks;
  kp.ksf_stride_h = kv_blocks * (p->D / 64) * 512;
  kp.ksf_stride_b = kp.ksf_stride_h * p->Hkv;
  // V scales: two 64-key column tiles per 128-key block, the last block padded with zeros
  kp.vsf_stride_h = (int64_t)((p->Dv + 127) / 128) * (2 * kv_blocks) * 512;
  kp.vsf_stride_b = kp.vsf_stride_h * p->Hkv;
  kp.seqused_k = cache.seqused_k;
  kp.page_table = cache.page_table;
  kp.page_size = cache.page_size;
  kp.pages_per_seq = cache.pages_per_seq;
  kp.cu_seqlens_q = cache.cu_seqlens_q;
  kp.cu_seqlens_k = cache.cu_seqlens_k;
  kp.cu_seqlens_v = cache.cu_seqlens_v;
  kp.total_q = cache.total_q;
  // Ranking the sequences costs 1-5 us at kernel start (grows with their number); it pays where long and
  // short ones are mixed.  us, slots / existing tiles: 24 sequences up to 2048 tokens 209 / 188, 4 up to 1500
  // 48 / 40; but 128 up to 300 36 / 38, 18 up to 142 17.8 / 20.
  kp.compact_tiles = cache.cu_seqlens_q != nullptr && p->B <= 256 && kp.num_m_blocks >= 8 &&
                     (int64_t)p->B * kp.num_m_blocks * 4 > 5 * ((int64_t)cache.total_q / kBlockM + p->B);
  kp.sl2 = p->softmax_scale * p->q_scale * p->k_scale * 1.4426950408889634f;
  kp.softcap_c1 = 0.f;
  if (softcap > 0.f) {
    // the kernel caps the raw products and then works in units of softcap * log2(e)
    kp.softcap_c1 = p->softmax_scale * p->q_scale * p->k_scale / softcap;
    kp.sl2 = softcap * 1.4426950408889634f;
  }
  kp.out_scale = p->v_scale;
  kp.q_scale = scales ? scales[0] : nullptr;
  kp.k_scale = scales ? scales[1] : nullptr;
  kp.v_scale = scales ? scales[2] : nullptr;
  kp.softmax_scale = p->softmax_scale;
  kp.softcap = softcap;
  kp.budget_ns = p->wait_budget_ns ? p->wait_budget_ns : kDefaultBudgetNs;
  kp.num_splits = num_splits;
  kp.Dv = p->Dv;
  kp.o_partial = static_cast<float*>(workspace);
  kp.lse_partial = workspace != nullptr
                       ? kp.o_partial + (int64_t)num_splits * p->B * p->Sq * p->Hq * p->Dv
                       : nullptr;

  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  const unsigned tiles = (unsigned)(kp.num_m_blocks * p->Hq * p->B * num_splits);
  kp.merge_splits = 0;
  bool merged = false;
  if (decode) {
    DecodeParams dp;
    dp.q = static_cast<const uint8_t*>(p->q);
    dp.q_sf = kp.q_sf;
    dp.q_stride_b = p->q_stride_b;
    dp.q_stride_s = p->q_stride_s;
    dp.q_stride_h = p->q_stride_h;
    dp.num_splits = num_splits;
    dp.o_partial = kp.o_partial;
    dp.lse_partial = kp.lse_partial;
    dp.lin = LinearScales{};
    if (linear != nullptr) {
      const int rows = cache.page_table ? cache.page_size : p->Sk;
      dp.lin = LinearScales{kp.q_sf, kp.k_sf, kp.v_sf, linear->q_stride_b, linear->q_stride_s, linear->q_stride_h,
                            linear->k_stride_b, linear->k_stride_s, linear->k_stride_h, linear->v_stride_b,
                            linear->v_stride_h, linear->v_stride_d, rows, (rows + 31) / 32 * 2};
    }
    const bool merge = decode_in_cluster(p, num_splits);
    dp.balance = Balance{};
    if (plan.balanced) {
      const int units = p->B * p->Hkv, slots = balanced_slots(p), ctas = balanced_ctas(p);
      dp.o_partial = static_cast<float*>(workspace);
      dp.lse_partial = dp.o_partial + (int64_t)ctas * dec_rows * 128;
      dp.balance = Balance{ctas, slots, dec::kMinBlocks, units >= kSortedUnits ? 6 : 1, 1.f / (float)slots,
                           1.f / (float)(ctas - units),
                           reinterpret_cast<int2*>(dp.lse_partial + ((int64_t)ctas * dec_rows + 3) / 4 * 4)};
      auto launch_bal = [&](auto kernel, int threads, uint32_t smem) -> int {
        return launch_pdl(kernel, dim3((unsigned)ctas), threads, smem, stream, tm_k, tm_v, kp, dp);
      };
#define FA4_DEC(rows, depth)                                                                                            \
  (linear != nullptr                                                                                                    \
       ? launch_bal(attn_decode_kernel<rows, kBalanced, depth, true>, dec::threads_of(rows, depth), dec::form<rows, depth>::kRequest) \
       : launch_bal(attn_decode_kernel<rows, kBalanced, depth, false>, dec::threads_of(rows, depth), dec::form<rows, depth>::kRequest))
      const int rc = dec_rows <= 4 ? FA4_DEC(4, 3) : dec_rows <= 8 ? FA4_DEC(8, 3) : dec_rows <= 16 ? FA4_DEC(16, 3) : FA4_DEC(32, 5);
#undef FA4_DEC
      if (rc != 0) return rc;
      const uint32_t rows = (uint32_t)(units * dec_rows);
      return launch_pdl(combine_pieces_kernel, dim3((rows + kCombineWarps - 1) / kCombineWarps), kCombineWarps * 32, 0, stream,
                        dp.o_partial, dp.lse_partial, dp.balance.pieces, kp.out, kp.lse, rows, dec_rows,
                        make_fastdiv((uint32_t)dec_rows), make_fastdiv((uint32_t)p->Hkv), kp.div_group, kp.Sq, kp.Hq, kp.Hkv, kp.group,
                        kp.o_stride_b, kp.o_stride_s, kp.o_stride_h);
    }
    auto launch_dec = [&](auto kernel, int threads, uint32_t smem) -> int {
      return launch_pdl_cluster(merge ? (unsigned)num_splits : 1u, kernel,
                                dim3((unsigned)num_splits, (unsigned)p->Hkv, (unsigned)p->B), threads, smem,
                                stream, tm_k, tm_v, kp, dp);
    };
    // The deep form where several entries have lengths of their own and no third CTA per SM waits: the long entries
    // then run on with few CTAs beside them, bound by the latency of their loads (paged batch of 16,
    // longest 8192: 23.9 -> 21.6 us before its four warpgroups, 18.6 with them).  Even lengths keep HBM busy with three
    // tiles, and the room beside two shallow CTAs lets the next call's start early (B=4, Sk=32768: 33.0 us shallow, 40.3
    // deep).
    // Not for clusters of three, five, six or seven, of which an SM's two places leave too few at once (one token, up to
    // 6528 keys, 8 heads: 5 entries in clusters of seven 12.8 us deep, 9.5 shallow; 6 in clusters of six 13.1, 10.3; 12 in
    // clusters of three 12.8, 9.9; but 16 entries of 2048 in pairs 8.8, 9.5).
    const bool deep = cache.seqused_k != nullptr && p->B >= 4 && (int64_t)num_splits * p->Hkv * p->B <= 2 * kSms &&
                      (!merge || (num_splits & (num_splits - 1)) == 0);
#define FA4_DEC_FORM(rows, merge, depth, linear)                                                      \
  launch_dec(attn_decode_kernel<rows, merge, depth, linear>, dec::threads_of(rows, depth), dec::form<rows, depth>::kRequest)
#define FA4_DEC(rows, depth)                                                                            \
  (linear != nullptr ? (merge ? FA4_DEC_FORM(rows, kCluster, depth, true) : FA4_DEC_FORM(rows, kWorkspace, depth, true)) \
                     : (merge ? FA4_DEC_FORM(rows, kCluster, depth, false) : FA4_DEC_FORM(rows, kWorkspace, depth, false)))
    const int rc = dec_rows <= 4    ? (deep ? FA4_DEC(4, 5) : FA4_DEC(4, 3))
                   : dec_rows <= 8  ? (deep ? FA4_DEC(8, 5) : FA4_DEC(8, 3))
                   : dec_rows <= 16 ? (deep ? FA4_DEC(16, 5) : FA4_DEC(16, 3))
                                    : FA4_DEC(32, 5);
#undef FA4_DEC
#undef FA4_DEC_FORM
    if (rc != 0 || merge) return rc;
  } else {
    // persistent: one CTA per SM walks the tile list
    int dev = 0, sms = 0;
    cudaError_t ce = cudaGetDevice(&dev);
    if (ce == cudaSuccess) ce = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (ce != cudaSuccess) return (int)ce;
    const unsigned grid = tiles < (unsigned)sms ? tiles : (unsigned)sms;
    CUtensorMap tm_o;
    {
      const bool packed = cache.cu_seqlens_q != nullptr;
      const uint64_t d_o[4] = {(uint64_t)p->Dv, (uint64_t)p->Hq, packed ? (uint64_t)cache.total_q : (uint64_t)p->Sq,
                               packed ? 1u : (uint64_t)p->B};
      const uint64_t s_o[3] = {(uint64_t)p->o_stride_h * 2, (uint64_t)p->o_stride_s * 2,
                               (uint64_t)p->o_stride_b * 2};
      // the 64-key kernel stores per warp (32 rows), the 128-key kernel a whole tile at a time
      if (!encode_out_4d(&tm_o, p->out, d_o, s_o, variant == FA4_VARIANT_WS64 ? 32u : 128u)) return -FA4_E_TENSORMAP;
    }
    auto launch = [&](auto kernel) -> int {
      if (int e = ensure_kernel(kernel, ws::kSmemRequest, ws::kRegsLaunch)) return e;
      // one work item per CTA and all clusters resident at once: the cluster of a tile merges its splits
      kp.merge_splits = num_splits > 1 && num_splits <= ws::kMaxCluster && tiles <= (unsigned)sms &&
                        clusters_at_once(reinterpret_cast<const void*>(kernel), num_splits, ws::kThreads,
                                         ws::kSmemRequest) * num_splits >= (int)tiles;
      merged = kp.merge_splits != 0;
      return launch_pdl_cluster(merged ? (unsigned)num_splits : 1u, kernel, dim3(grid), ws::kThreads, ws::kSmemRequest, stream, tm_q, tm_k, tm_v, tm_o, kp);
    };
    int rc;
    if (variant == FA4_VARIANT_WS64) {
      auto launch64 = [&](auto kernel) -> int {
        if (int e = ensure_kernel(kernel, ws64::kSmemRequest, ws64::kRegsLaunch)) return e;
        // as many launches as the per-CTA tile table asks for (one up to 113 664 tiles on 148 SMs)
        for (uint32_t begin = 0; begin < tiles; begin += grid * ws64::kMaxTiles) {
          kp.tile_begin = (int)begin;
          kp.tile_end = (int)(tiles - begin < grid * ws64::kMaxTiles ? tiles : begin + grid * ws64::kMaxTiles);
          if (int e = launch_pdl(kernel, dim3(grid), ws64::kThreads, ws64::kSmemRequest, stream, tm_q, tm_k, tm_v, tm_o, kp))
            return e;
        }
        return 0;
      };
      // Windows of up to two blocks' worth of keys run the narrow form of the kernel.  us at B=2, S=4096,
      // Hq=32, Hkv=8, causal, wide form / narrow form, D = 128: 64 keys 51.7/45.4, 128 54.1/49.2, 192 57.5/57.8, 256
      // 59.6/58.1, 288 67.6/68.2, 384 63.8/64.7, 512 72.7/74.1.  D = 64: 128 44.8/40.4, 256 51.4/49.6, 384 59.2/55.8, 512
      // 68.0/66.0; D = 192: 57.2/50.7, 63.3/57.7, 65.2/61.2, 73.4/70.9 (there the narrow form is ahead beyond the line too,
      // by 3-6 %).
      const bool narrow = win_left >= 0 && win_right >= 0 && (int64_t)win_left + win_right <= 256;
#define FA4_WS64(...)                                                                                     \
  (p->D == 128 ? launch64(attn_fwd_ws64_kernel<128, __VA_ARGS__>)                                        \
               : (p->D == 64 ? launch64(attn_fwd_ws64_kernel<64, __VA_ARGS__>) : launch64(attn_fwd_ws64_kernel<192, __VA_ARGS__>)))
      // The soft cap has its own instantiations: 64 tanh and selects in the middle of the loop are 6 KB of code, a
      // fifth of what an SM's instruction cache holds (24 packed sequences up to 2048, no cap: 174 us with the code in
      // the kernel, 168 without).
      const bool cap = softcap > 0.f;
      if (general && local && narrow)           // window (with or without sink / cache view)
        rc = cap ? FA4_WS64(true, true, true, true, true) : FA4_WS64(true, true, true, true);
      else if (general && local)
        rc = cap ? FA4_WS64(true, true, true, false, true) : FA4_WS64(true);
      else if (general && cached)               // KV-cache view without a window
        rc = cap ? FA4_WS64(true, false, true, false, true) : FA4_WS64(true, false, true);
      else if (general)                         // sink / soft cap only: plain tile geometry
        rc = cap ? FA4_WS64(true, false, false, false, true) : FA4_WS64(true, false);
      else
        rc = FA4_WS64(false);
#undef FA4_WS64
    } else if (p->D == 128) {
      rc = !general ? launch(attn_fwd_ws_kernel<128, false>)
                    : (local ? launch(attn_fwd_ws_kernel<128, true>)
                             : (softcap > 0.f ? launch(attn_fwd_ws_kernel<128, true, false>)
                                              : launch(attn_fwd_ws_kernel<128, true, false, false>)));
    } else {
      rc = !general ? launch(attn_fwd_ws_kernel<64, false>)
                    : (local ? launch(attn_fwd_ws_kernel<64, true>)
                             : (softcap > 0.f ? launch(attn_fwd_ws_kernel<64, true, false>)
                                              : launch(attn_fwd_ws_kernel<64, true, false, false>)));
    }
    if (rc != 0) return rc;
  }
  if ((num_splits > 1 || decode) && !merged) {
    // (fewer than 2^31 rows: the workspace holds at least 512 bytes of each)
    const uint32_t rows = (uint32_t)p->B * p->Sq * p->Hq;
    const bool shared_rows = num_splits > kCombineBatch && rows <= kCombineSharedRows;
    const uint32_t per_block = shared_rows ? 1u : kCombineWarps * 128u / (uint32_t)p->Dv;
    uint32_t blocks = (rows + per_block - 1) / per_block;
    if (blocks > kSms * kCombineBlocksPerSm) blocks = kSms * kCombineBlocksPerSm;
    return launch_pdl(combine_splits_kernel, dim3(blocks), kCombineWarps * 32, 0, stream, kp.o_partial, kp.lse_partial,
                      kp.out, kp.lse, num_splits, rows, shared_rows ? kCombineWarps : 1, kp.div_hq,
                      make_fastdiv((uint32_t)p->Sq), p->Sq, p->Hq, p->Dv, kp.o_stride_b, kp.o_stride_s, kp.o_stride_h);
  }
  return 0;
}
}  // namespace

extern "C" int fa4_nvfp4_sf_linear_to_tiled(const void* src, void* dst, int32_t n_outer,
                                            int32_t n_inner, int32_t rows, int32_t cols,
                                            int64_t stride_outer, int64_t stride_inner,
                                            int64_t stride_row, int32_t col_tile_multiple,
                                            void* cuda_stream) {
  const fa4_nvfp4_sf_job j = {src, dst, nullptr, n_outer, n_inner, rows, cols, stride_outer, stride_inner, stride_row,
                              col_tile_multiple, 0};
  return fa4_nvfp4_sf_tile_jobs(&j, 1, cuda_stream);
}

// ---------------------------------------------------------------------------------------------
// Fused NVFP4 quantiser (bf16 operands in the reference layout -> what fa4_nvfp4_fwd reads)
// ---------------------------------------------------------------------------------------------
namespace {
constexpr int64_t kMaxQuantUnits = 0x7fffffffll;

// Number of CTAs of a tensor that has `units` of `total` units of work, at most one per `per_cta` units.
int share_of(int64_t ctas, int64_t units, int64_t total, int64_t per_cta) {
  const int64_t want = (ctas * units + total - 1) / total, most = (units + per_cta - 1) / per_cta;
  return (int)(want < 1 ? 1 : (want < most ? want : most));
}

// Shape, strides and alignment of one tensor; the fields of the amax pass.
int describe_tensor(QuantJob* j, const void* x, int64_t B, int64_t S, int64_t H, int64_t D, int64_t sb, int64_t ss,
                    int64_t sh) {
  if (!x) return -FA4_E_NULL;
  if (B <= 0 || S <= 0 || H <= 0 || D <= 0 || D % 8 != 0) return -FA4_E_SHAPE;
  if (sb % 8 != 0 || ss % 8 != 0 || sh % 8 != 0) return -FA4_E_STRIDE;
  if (!aligned16(x)) return -FA4_E_ALIGN;
  if (B > 0x7fffffffll || S > 0x7fffffffll || H > 0x7fffffffll || D > 0x7fffffffll) return -FA4_E_TOO_LARGE;
  *j = QuantJob{};
  j->x = static_cast<const __nv_bfloat16*>(x);
  j->sb = sb; j->ss = ss; j->sh = sh;
  j->B = (int)B; j->S = (int)S; j->H = (int)H; j->D = (int)D;
  j->wide = ((reinterpret_cast<uintptr_t>(x) | (uintptr_t)(2 * (sb | ss | sh | D))) & 31u) == 0;
  // the tensor as runs of contiguous elements, merged as far as the strides allow
  int64_t inner = D, n0 = B, n1 = S, n2 = H, r0 = sb, r1 = ss, r2 = sh;
  auto merge = [&](int64_t n, int64_t stride) { return n == 1 || stride == inner; };
  if (merge(H, sh)) {
    inner *= H; n0 = 1; n1 = B; n2 = S; r0 = 0; r1 = sb; r2 = ss;
    if (merge(S, ss)) {
      inner *= S; n1 = 1; n2 = B; r1 = 0; r2 = sb;
      if (merge(B, sb)) { inner *= B; n2 = 1; r2 = 0; }
    }
  }
  j->unit = inner % 16 == 0 ? 16 : 8;
  const int64_t units = n0 * n1 * n2 * (inner / j->unit);
  if (units > kMaxQuantUnits) return -FA4_E_TOO_LARGE;
  j->units = (uint32_t)units;
  j->inner_units = (int)(inner / j->unit);
  j->n1 = (int)n1; j->n2 = (int)n2;
  j->r0 = r0; j->r1 = r1; j->r2 = r2;
  j->div_inner = make_fastdiv((uint32_t)j->inner_units);
  j->div_n2 = make_fastdiv((uint32_t)n2);
  j->div_n1 = make_fastdiv((uint32_t)n1);
  return 0;
}

// The fields of the quantise pass.
int describe_outputs(QuantJob* j, bool is_v, int64_t s_out, void* packed, void* sf_linear, void* sf_tiled, float* scale_out) {
  if (!packed) return -FA4_E_NULL;
  if (!aligned16(packed) || (sf_linear && !aligned16(sf_linear)) || (sf_tiled && !aligned16(sf_tiled))) return -FA4_E_ALIGN;
  j->is_v = is_v;
  j->packed = static_cast<uint8_t*>(packed);
  j->lin = static_cast<uint8_t*>(sf_linear);
  j->tiled = static_cast<uint8_t*>(sf_tiled);
  j->scale_out = scale_out;
  int64_t items;
  if (is_v) {
    if (s_out < j->S || s_out % 16 != 0 || s_out > 0x7fffffffll) return -FA4_E_SHAPE;
    j->s_out = (int)s_out;
    j->rt = (int)((s_out + 127) / 128);
    items = (int64_t)j->B * j->H * ((j->D + 127) / 128) * j->rt;
    j->div_h = make_fastdiv((uint32_t)j->H);
  } else {
    if (j->D % 64 != 0) return -FA4_E_SHAPE;
    j->nb = j->H * (j->D / 16);
    j->rt = (j->S + 127) / 128;
    items = (int64_t)j->B * j->rt * 32 * j->nb;
    // four rows per item once that gives every SM its CTAs
    j->single = items < kSms * kQuantizeCtas * 256;
    if (j->single) items *= 4;
    j->div_nb = make_fastdiv((uint32_t)j->nb);
    j->div_h = make_fastdiv((uint32_t)(j->D / 16));
  }
  if (items > kMaxQuantUnits) return -FA4_E_TOO_LARGE;
  j->items = (uint32_t)items;
  j->div_rt = make_fastdiv((uint32_t)j->rt);
  return 0;
}

int launch_amax(QuantJobs& q, cudaStream_t stream) {
  int64_t total = 0;
  int blocks = 0;
  for (int i = 0; i < q.n; ++i) total += q.job[i].units;
  for (int i = 0; i < q.n; ++i) {
    QuantJob& j = q.job[i];
    j.amax_block0 = blocks;
    j.amax_blocks = share_of(kSms * kAmaxCtas, j.units, total, kAmaxThreads);
    j.parts = q.parts + blocks;
    j.num_parts = j.amax_blocks;
    blocks += j.amax_blocks;
  }
  return launch_pdl(amax_kernel, dim3(blocks), kAmaxThreads, 0, stream, q);
}

int launch_quantize(QuantJobs& q, cudaStream_t stream) {
  // bytes, V's weighted by what its transpose costs more
  auto weight = [](const QuantJob& j) { return (int64_t)j.units * j.unit * (j.is_v ? kQuantizeVWeight : 16); };
  int64_t total = 0, blocks = 0;
  for (int i = 0; i < q.n; ++i) total += weight(q.job[i]);
  for (int i = 0; i < q.n; ++i) {
    QuantJob& j = q.job[i];
    const int64_t most = j.is_v ? j.items : ((int64_t)j.items + 255) / 256;
    int64_t ctas = kSms * kQuantizeCtas * weight(j) / total;
    if (ctas < 1) ctas = 1;
    if (ctas > most || j.single) ctas = most;
    j.block0 = (int)blocks;
    j.blocks = (int)ctas;
    blocks += ctas;
  }
  return launch_pdl(quantize_kernel, dim3((unsigned)blocks), 256, kQuantizeSmem, stream, q);
}
}  // namespace

extern "C" int fa4_nvfp4_quantize_jobs_bf16(const fa4_nvfp4_quant_job* jobs, int32_t n, float* scratch, void* cuda_stream) {
  if (!jobs || !scratch) return -FA4_E_NULL;
  if (n < 1 || n > 3) return -FA4_E_SHAPE;
  QuantJobs q{};
  q.n = n;
  q.parts = scratch;
  for (int i = 0; i < n; ++i) {
    const fa4_nvfp4_quant_job& a = jobs[i];
    if (int e = describe_tensor(&q.job[i], a.x, a.B, a.S, a.H, a.D, a.stride_b, a.stride_s, a.stride_h)) return e;
    if (int e = describe_outputs(&q.job[i], a.is_v != 0, a.S_out, a.packed, a.sf_linear, a.sf_tiled, a.scale_out)) return e;
  }
  const cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  if (int e = launch_amax(q, stream)) return e;
  return launch_quantize(q, stream);
}

extern "C" int fa4_nvfp4_amax_bf16(const void* x, int64_t n0, int32_t n1, int32_t n2, int32_t inner,
                                   int64_t s0, int64_t s1, int64_t s2, float* amax,
                                   void* cuda_stream) {
  if (!amax) return -FA4_E_NULL;
  QuantJobs q{};
  q.n = 1;
  if (int e = describe_tensor(&q.job[0], x, n0, n1, n2, inner, s0, s1, s2)) return e;
  q.job[0].amax_out = amax;
  return launch_amax(q, static_cast<cudaStream_t>(cuda_stream));
}

namespace {
int quantize_with_amax(const void* x, bool is_v, int32_t B, int32_t S, int32_t H, int32_t D, int64_t sb, int64_t ss,
                       int64_t sh, const float* amax, void* packed, void* sf_linear, void* sf_tiled, float* scale_out,
                       void* cuda_stream) {
  if (!amax) return -FA4_E_NULL;
  QuantJobs q{};
  q.n = 1;
  if (int e = describe_tensor(&q.job[0], x, B, S, H, D, sb, ss, sh)) return e;
  if (int e = describe_outputs(&q.job[0], is_v, S, packed, sf_linear, sf_tiled, scale_out)) return e;
  q.job[0].parts = amax;
  q.job[0].num_parts = 1;
  return launch_quantize(q, static_cast<cudaStream_t>(cuda_stream));
}
}  // namespace

extern "C" int fa4_nvfp4_quantize_qk_bf16(const void* x, int32_t B, int32_t S, int32_t H, int32_t D,
                                          int64_t stride_b, int64_t stride_s, int64_t stride_h,
                                          const float* amax, void* packed, void* sf_linear,
                                          void* sf_tiled, float* scale_out, void* cuda_stream) {
  return quantize_with_amax(x, false, B, S, H, D, stride_b, stride_s, stride_h, amax, packed, sf_linear, sf_tiled,
                            scale_out, cuda_stream);
}

extern "C" int fa4_nvfp4_quantize_v_bf16(const void* x, int32_t B, int32_t Sk, int32_t H, int32_t Dv,
                                         int64_t stride_b, int64_t stride_s, int64_t stride_h,
                                         const float* amax, void* packed, void* sf_linear,
                                         void* sf_tiled, float* scale_out, void* cuda_stream) {
  return quantize_with_amax(x, true, B, Sk, H, Dv, stride_b, stride_s, stride_h, amax, packed, sf_linear, sf_tiled,
                            scale_out, cuda_stream);
}

extern "C" int fa4_nvfp4_debug_qk_tile(const void* q, const void* k, const void* q_sf,
                                       const void* k_sf, float* s_out, int32_t D, int32_t mode,
                                       uint32_t* status, void* cuda_stream) {
  if (!q || !k || !q_sf || !k_sf || !s_out) return -FA4_E_NULL;
  if (D != 128) return -FA4_E_SHAPE;
  if (!aligned16(q) || !aligned16(k) || !aligned16(q_sf) || !aligned16(k_sf)) return -FA4_E_ALIGN;
  CUtensorMap tm_q, tm_k;
  const uint64_t d[4] = {64, 1, 128, 1};
  const uint64_t s[3] = {64, 64, 64 * 128};
  const uint32_t b[4] = {64, 1, 128, 1};
  if (!encode_u8_4d(&tm_q, q, d, s, b, CU_TENSOR_MAP_SWIZZLE_64B) ||
      !encode_u8_4d(&tm_k, k, d, s, b, CU_TENSOR_MAP_SWIZZLE_64B))
    return -FA4_E_TENSORMAP;
  if (int e = ensure_smem(qk_tile_probe_kernel, kProbeSmemRequest)) return e;
  qk_tile_probe_kernel<<<1, 128, kProbeSmemRequest, static_cast<cudaStream_t>(cuda_stream)>>>(
      tm_q, tm_k, static_cast<const uint8_t*>(q), static_cast<const uint8_t*>(k),
      static_cast<const uint8_t*>(q_sf), static_cast<const uint8_t*>(k_sf), s_out, mode, status,
      kDefaultBudgetNs);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : (int)e;
}

extern "C" int fa4_nvfp4_debug_mma_rate(int32_t iters, int32_t num_ctas, uint64_t* clocks_out,
                                        uint32_t* status, void* cuda_stream) {
  if (!clocks_out) return -FA4_E_NULL;
  if (iters < 4 || iters % 4 != 0 || iters > (1 << 22) || num_ctas < 1 || num_ctas > 1024)
    return -FA4_E_SHAPE;
  if (int e = ensure_smem(mma_rate_kernel, kProbeSmemRequest)) return e;
  mma_rate_kernel<<<num_ctas, 128, kProbeSmemRequest, static_cast<cudaStream_t>(cuda_stream)>>>(
      iters, reinterpret_cast<unsigned long long*>(clocks_out), status, kDefaultBudgetNs);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : (int)e;
}

extern "C" int fa4_nvfp4_debug_ex2_rate(int32_t iters, int32_t num_ctas, uint64_t* clocks_out, float* scratch,
                                        void* cuda_stream) {
  if (!clocks_out || !scratch) return -FA4_E_NULL;
  if (iters < 1 || iters > (1 << 22) || num_ctas < 1 || num_ctas > 1024) return -FA4_E_SHAPE;
  ex2_rate_kernel<<<num_ctas, 512, 0, static_cast<cudaStream_t>(cuda_stream)>>>(
      iters, reinterpret_cast<unsigned long long*>(clocks_out), scratch);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : (int)e;
}

extern "C" int fa4_nvfp4_debug_wait_expiry(uint32_t* status, uint64_t budget_ns, void* cuda_stream) {
  if (!status) return -FA4_E_NULL;
  if (budget_ns == 0 || budget_ns > kDefaultBudgetNs) return -FA4_E_SHAPE;
  wait_expiry_kernel<<<1, 32, 0, static_cast<cudaStream_t>(cuda_stream)>>>(status, budget_ns);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : (int)e;
}

// ---------------------------------------------------------------------------------------------
// Forward from LINEAR scale factors without any allocation.
//
// The regular route for linear scale factors needs scratch memory: three tiled copies of the
// scales that the caller (the Python wrapper) allocates before calling
// fa4_nvfp4_sf_linear_to_tiled and fa4_nvfp4_fwd.  Some hosts cannot do that: a serving
// process that handed every byte of device memory to its own arena at start-up, or a
// steady-state loop that runs under a "no cudaMalloc" rule because the call synchronises the
// device.  For them the scratch lives in the library image instead: one fixed array per GPU,
// resident from the moment the library is loaded on that GPU until the process exits.
//
// The array name below is only a host-side handle; every call asks the runtime for the device
// address on the current device (cudaGetSymbolAddress), so a pointer from before a
// cudaDeviceReset is never reused.
// ---------------------------------------------------------------------------------------------
#define FA4_STATIC_SCRATCH_BYTES (16u << 20)
static __device__ __align__(256) uint8_t g_sf_scratch[FA4_STATIC_SCRATCH_BYTES];

namespace {
inline int64_t tiled_sf_bytes(int64_t n_mats, int64_t rows, int64_t cols, int64_t ct_multiple) {
  const int64_t ct = ((cols + 3) / 4 + ct_multiple - 1) / ct_multiple * ct_multiple;
  return n_mats * ((rows + 127) / 128) * ct * 512;
}
}  // namespace

extern "C" int fa4_nvfp4_fwd_linear_sf_noalloc(const fa4_nvfp4_params* p, void* cuda_stream) {
  // 1. every host-side check of the forward itself, before anything touches the GPU or the
  //    shared array: a negative return means nothing was launched and nothing was overwritten
  FwdPlan plan;
  if (int e = validate_fwd(p, 1, nullptr, 0, -1, -1, nullptr, 0.f, CacheView{}, /*linear_sf=*/true, &plan))
    return e;
  if (plan.variant == FA4_VARIANT_DECODE) return -FA4_E_VARIANT;   // needs a caller-owned workspace
  // 2. capacity of the array
  const int64_t q_bytes = tiled_sf_bytes((int64_t)p->B * p->Hq, p->Sq, p->D / 16, 1);
  const int64_t k_bytes = tiled_sf_bytes((int64_t)p->B * p->Hkv, p->Sk, p->D / 16, 1);
  const int64_t skp = ((int64_t)p->Sk + 31) / 32 * 32;   // V's padded key axis
  const int64_t v_bytes = tiled_sf_bytes((int64_t)p->B * p->Hkv, p->Dv, skp / 16, 2);
  if (q_bytes + k_bytes + v_bytes > (int64_t)FA4_STATIC_SCRATCH_BYTES) return -FA4_E_TOO_LARGE;

  // 3. device address of the array on the current device
  void* sym = nullptr;
  const cudaError_t se = cudaGetSymbolAddress(&sym, g_sf_scratch);
  if (se != cudaSuccess) return (int)se;
  uint8_t* q_t = static_cast<uint8_t*>(sym);
  uint8_t* k_t = q_t + q_bytes;   // multiples of 512: every region stays 256-byte aligned
  uint8_t* v_t = k_t + k_bytes;

  const int64_t cq = p->D / 16, cv = skp / 16;
  // q_sf (B, Sq, Hq, D/16) and k_sf (B, Sk, Hkv, D/16): matrix (b, h) has row stride H * D/16;
  // v_sf (B, Hkv, Dv, Sk/16): matrix (b, h) is contiguous
  const fa4_nvfp4_sf_job jobs[3] = {
      {p->q_sf, q_t, nullptr, p->B, p->Hq, p->Sq, (int32_t)cq, p->Sq * p->Hq * cq, cq, p->Hq * cq, 1, 0},
      {p->k_sf, k_t, nullptr, p->B, p->Hkv, p->Sk, (int32_t)cq, p->Sk * p->Hkv * cq, cq, p->Hkv * cq, 1, 0},
      {p->v_sf, v_t, nullptr, p->B, p->Hkv, p->Dv, (int32_t)cv, p->Hkv * p->Dv * cv, p->Dv * cv, cv, 2, 0}};
  if (int e = fa4_nvfp4_sf_tile_jobs(jobs, 3, cuda_stream)) return e;
  fa4_nvfp4_params tiled = *p;
  tiled.q_sf = q_t;
  tiled.k_sf = k_t;
  tiled.v_sf = v_t;
  return fa4_nvfp4_fwd(&tiled, cuda_stream);
}
