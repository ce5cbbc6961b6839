// Fused NVFP4 quantiser of the attention operands: bf16 -> packed e2m1 + ue4m3 block scales
// (linear and / or the tiled layout the attention kernel reads) in one pass over the tensor,
// after one amax pass.  The step directly in front of the attention forward; the reference has
// no quantiser for this path (flash_attn/cute/interface.py:370 rejects anything but fp16/bf16).
//
// Arithmetic (identical, bit for bit, to the CPU oracle's quantize_nvfp4):
//   tensor scale g = amax / (6 * 448)                      (1 when the tensor is all zero)
//   block scale    = e4m3_rne(min((block amax / 6) / g, 448))          per 16 elements
//   element        = e2m1_rne(x / (float(block scale) * g)), no negative zero
// every operation a correctly rounded fp32 one.
//
// Two launches for the q, k and v of a call (any one to three tensors): amax_kernel writes one partial
// maximum per CTA, quantize_kernel reduces them and quantises.  2 B read per element in each pass,
// 9/16 B (10/16 with both scale layouts) written: HBM-bound byte movers.  The second pass walks every
// tensor from its end, where the first pass has just been, so that its first tens of MB come from L2.
#pragma once
#include "ptx.cuh"
#include <cuda_bf16.h>

namespace fa4 {

__device__ __forceinline__ float tensor_scale_of(float amax) {
  return amax > 0.f ? __fdiv_rn(amax, 6.f * 448.f) : 1.f;
}

// ue4m3 byte of a non-negative fp32 (round to nearest even, saturating at 448).
__device__ __forceinline__ uint32_t e4m3_byte(float v) {
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(0.f), "f"(v));
  return r & 0xffu;
}
__device__ __forceinline__ float e4m3_value(uint32_t byte) {
  uint32_t h2;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"(static_cast<uint16_t>(byte)));
  return __half2float(__ushort_as_half(static_cast<unsigned short>(h2 & 0xffffu)));
}

// Clears the sign of nibbles whose magnitude is zero (the formats agree on "no negative zero"): a magnitude
// of 1..7 plus 7 sets bit 3 of its nibble and carries no further.
__device__ __forceinline__ uint32_t drop_negative_zero(uint32_t n) {
  return n & (((n & 0x77777777u) + 0x77777777u) | 0x77777777u);
}

// a / b from 1 / b in two terms, hi + lo (lo = the residual of hi, times hi): the product is within a few
// 2^-47 of the quotient before its one rounding.  That is not always the correctly rounded quotient, but
// on the same side of every rounding boundary that matters here, for every a and b that can occur
// (tests/test_quantiser_rounding_cpu.py goes through all of them).  Two FMA-pipe instructions; needs lo to be no
// denormal, so callers keep b between 1e-30 and 1e20.
struct Reciprocal {
  float hi, lo;
};
__device__ __forceinline__ float div_by(float a, const Reciprocal& r) { return fmaf(a, r.hi, __fmul_rn(a, r.lo)); }

// Rare path of quantize_block16 (denominators near the bottom of the fp32 range), out of line so
// that the hot loop stays small.
struct Block16 {
  float v[16];
};
__device__ __noinline__ uint2 quantize_block16_exact(Block16 x, float denom) {
  float y[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) y[i] = denom > 0.f ? __fdiv_rn(x.v[i], denom) : 0.f;
  return make_uint2(pack8_e2m1(y[0], y[1], y[2], y[3], y[4], y[5], y[6], y[7]),
                    pack8_e2m1(y[8], y[9], y[10], y[11], y[12], y[13], y[14], y[15]));
}

// Per-tensor constants of the quantiser: the tensor scale g, 1 / g, and whether g or a block's scale times g lies
// where the two-term reciprocals lose bits (`odd`: block scales take the library division; `exact`: the elements
// as well).  That is near the ends of the fp32 range, and where the significand of such a product is all ones: no bf16 maximum
// gives one, but a caller's own may, and the reciprocal of 2 - 2^-23 is one ulp too small: the quotient of .5 is then on the
// boundary .25 instead of above it.
struct TensorScale {
  float g;
  Reciprocal rcp;
  bool odd, exact, finite;
};
__device__ __forceinline__ TensorScale make_tensor_scale(float amax) {
  TensorScale t;
  t.g = tensor_scale_of(amax);
  bool ones = false;           // (an e4m3 value has four bits)
#pragma unroll
  for (int m = 8; m < 16; ++m) ones |= (~__float_as_uint(__fmul_rn((float)m, t.g)) & 0x7fffffu) == 0u;
  t.exact = (t.g > 1e17f && t.g < INFINITY) || ones;
  t.odd = !(t.g >= 1e-18f) || t.exact;
  t.finite = t.g < INFINITY;
  t.rcp.hi = t.odd ? 0.f : __frcp_rn(t.g);
  t.rcp.lo = fmaf(-t.g, t.rcp.hi, 1.f) * t.rcp.hi;
  return t;
}

// Scale byte and its value times g for a block with maximum bmax.
__device__ __forceinline__ float block_scale_of(float bmax, const TensorScale& ts, uint32_t& sf_byte) {
  // block scale = e4m3_rne(min((bmax / 6) / g, 448)).  With g >= 1e-18 every quotient that can
  // reach the first rounding boundary of e4m3 (2^-10) is far from the denormals; smaller quotients give
  // the zero byte whatever their last bits are.
  constexpr float kSixth = 0.16666667163372039794921875f;   // RN(1 / 6), and 1 / 6 minus it
  constexpr Reciprocal kRcp6 = {kSixth, -4.967053731282552e-09f};
  float t;
  if (ts.odd) {
    t = __fdiv_rn(__fdiv_rn(bmax, 6.f), ts.g);
  } else {
    t = div_by(div_by(bmax, kRcp6), ts.rcp);
  }
  sf_byte = e4m3_byte(fminf(t, 448.f));
  return __fmul_rn(e4m3_value(sf_byte), ts.g);
}

// One block of 16 values with maximum bmax -> 8 packed bytes (two words) and its scale byte.
__device__ __forceinline__ void quantize_block16(const float (&x)[16], float bmax, const TensorScale& ts,
                                                 uint32_t& lo, uint32_t& hi, uint32_t& sf_byte) {
  const float denom = block_scale_of(bmax, ts, sf_byte);
  // The element codes are those of the correctly rounded quotients x / denom: only quotients within a few
  // ulp of a rounding boundary of e2m1 (.25 .75 1.25 1.75 2.5 3.5 5) matter, x has eight significand bits, and
  // for every significand of denom but the largest (which takes the other branch) and every reciprocal
  // within one ulp the products below put the values of x next to a boundary on the side of it that the
  // correctly rounded quotient is on.  Two instructions a pair where one term and a residual step took three.
  // An infinity in front of a residual of either sign would be an infinity or a NaN: with a tensor scale that leaves it a
  // value (a caller's own), the block takes the quotients.
  if (denom >= 1e-30f && !ts.exact && (bmax < INFINITY || !ts.finite)) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(denom));
    const float rl = __fmul_rn(fmaf(-denom, r, 1.f), r);
    const float2 r2 = make_float2(r, r), rl2 = make_float2(rl, rl);
    float2 y[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 v = make_float2(x[2 * i], x[2 * i + 1]);
      y[i] = __ffma2_rn(v, r2, __fmul2_rn(v, rl2));
    }
    lo = pack8_e2m1(y[0].x, y[0].y, y[1].x, y[1].y, y[2].x, y[2].y, y[3].x, y[3].y);
    hi = pack8_e2m1(y[4].x, y[4].y, y[5].x, y[5].y, y[6].x, y[6].y, y[7].x, y[7].y);
  } else {
    Block16 blk;
#pragma unroll
    for (int i = 0; i < 16; ++i) blk.v[i] = x[i];
    const uint2 e = quantize_block16_exact(blk, denom);
    lo = e.x;
    hi = e.y;
  }
  lo = drop_negative_zero(lo);
  hi = drop_negative_zero(hi);
}


// 32 consecutive bytes of global memory: one 256-bit load when the address allows it
struct Words8 {
  uint32_t w[8];
};
__device__ __forceinline__ Words8 load32(const void* p, bool wide) {
  Words8 v;
  if (wide) {
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]), "=r"(v.w[4]), "=r"(v.w[5]), "=r"(v.w[6]),
                   "=r"(v.w[7])
                 : "l"(p));
  } else {
    const uint4 a = *static_cast<const uint4*>(p), b = *(static_cast<const uint4*>(p) + 1);
    v.w[0] = a.x; v.w[1] = a.y; v.w[2] = a.z; v.w[3] = a.w;
    v.w[4] = b.x; v.w[5] = b.y; v.w[6] = b.z; v.w[7] = b.w;
  }
  return v;
}
// max(|a|, |b|) of two bf16 pairs (a NaN loses to a number, like fmaxf); the result's signs are noise
__device__ __forceinline__ uint32_t absmax2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ float max_of_pair(uint32_t m) {
  return fmaxf(fabsf(__uint_as_float(m << 16)), fabsf(__uint_as_float(m & 0xffff0000u)));
}
__device__ __forceinline__ float absmax16(const Words8& v) {
  return max_of_pair(absmax2(absmax2(absmax2(v.w[0], v.w[1]), absmax2(v.w[2], v.w[3])),
                             absmax2(absmax2(v.w[4], v.w[5]), absmax2(v.w[6], v.w[7]))));
}

// One tensor of a launch: bf16 (B, S, H, D), last dimension contiguous.
struct QuantJob {
  const __nv_bfloat16* x;
  int64_t sb, ss, sh;           // strides in elements
  int B, S, H, D;
  int s_out;                    // V: its key axis as stored (zeros from S on)
  int is_v, wide;               // wide: every 32-byte piece is 32-byte aligned
  // amax pass: units of 16 elements (8 where a run is no multiple of 16); the tensor as (n0, n1, n2)
  // runs of inner_units
  uint32_t units;
  int unit;
  int amax_block0, amax_blocks;
  int64_t r0, r1, r2;           // strides of the runs
  FastDiv div_inner, div_n2, div_n1;
  int inner_units, n2, n1;
  float* amax_out;              // atomic maximum of the tensor (then no partials), or null
  // quantise pass
  const float* parts;           // partial maxima of this tensor
  int num_parts;
  int block0, blocks;
  int single;                   // Q / K: one row per work item instead of four (tensors too small to fill the GPU)
  uint32_t items;               // Q / K: threads' work items; V: tiles
  FastDiv div_nb, div_rt, div_h;
  int nb, rt;                   // Q / K: blocks of a row of all heads; 128-row (V: 128-key) tiles
  uint8_t *packed, *lin, *tiled;
  float* scale_out;
};
struct QuantJobs {
  QuantJob job[3];
  float* parts;                 // amax pass: one float per CTA of the grid
  int n;
};

// ---------------------------------------------------------------------------------------------
// Partial maxima of |x|, one per CTA (or an atomicMax into amax_out, bit patterns of values >= 0).
// Two 32-byte loads in flight per thread, 1536 threads per SM: q, k, v of B=4, S=8192, Hq=32, Hkv=8, D=128
// in 70 us (5.7 TB/s).  Four loads and 2048 threads in larger CTAs: 80; eight: 86 (the CTAs then
// spread over too many DRAM pages at a time).  The three launches it replaced: 97.
// ---------------------------------------------------------------------------------------------
constexpr int kAmaxThreads = 256, kAmaxCtas = 6;   // CTAs per SM
__global__ void __launch_bounds__(kAmaxThreads)
amax_kernel(const __grid_constant__ QuantJobs jobs) {
  __shared__ float warp_max[kAmaxThreads / 32];
  pdl_wait();
  int ji = 0;
  while (ji + 1 < jobs.n && (int)blockIdx.x >= jobs.job[ji + 1].amax_block0) ++ji;
  const QuantJob& j = jobs.job[ji];
  const uint32_t stride = (uint32_t)j.amax_blocks * kAmaxThreads;
  const bool flat = j.n1 * j.n2 == 1 && j.inner_units >= (int)j.units, wide = j.wide != 0;
  auto at = [&](uint32_t u) -> const __nv_bfloat16* {
    if (flat) return j.x + (int64_t)u * j.unit;
    const int run = fast_div((int)u, j.div_inner), c = (int)u - run * j.inner_units;
    const int i01 = fast_div(run, j.div_n2), i2 = run - i01 * j.n2;
    const int i0 = fast_div(i01, j.div_n1), i1 = i01 - i0 * j.n1;
    return j.x + i0 * j.r0 + i1 * j.r1 + i2 * j.r2 + (int64_t)c * j.unit;
  };
  const bool half = j.unit == 8;
  auto load = [&](uint32_t i) -> Words8 {
    if (!half) return load32(at(i), wide);
    const uint4 a = *reinterpret_cast<const uint4*>(at(i));
    return Words8{{a.x, a.y, a.z, a.w, 0u, 0u, 0u, 0u}};
  };
  uint32_t m2 = 0u;
  uint32_t u = (blockIdx.x - j.amax_block0) * kAmaxThreads + threadIdx.x;
  for (; u + (uint64_t)stride < j.units; u += 2 * stride) {
    Words8 v[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) v[k] = load(u + k * stride);
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int i = 0; i < 8; ++i) m2 = absmax2(m2, v[k].w[i]);
  }
  for (; u < j.units; u += stride) {
    const Words8 v = load(u);
#pragma unroll
    for (int i = 0; i < 8; ++i) m2 = absmax2(m2, v.w[i]);
  }
  float m = max_of_pair(m2);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < kAmaxThreads / 32; ++w) m = fmaxf(m, warp_max[w]);
    if (j.amax_out == nullptr) jobs.parts[blockIdx.x] = m;
    else if (m > 0.f) atomicMax(reinterpret_cast<int*>(j.amax_out), __float_as_int(m));
  }
}

// ---------------------------------------------------------------------------------------------
// Quantise.  CTAs are dealt to the tensors in proportion to their size and walk them from the end.
//
// Q / K, blocks along D: a work item is one block of 16 in the rows l, l + 32, l + 64, l + 96 of a
// 128-row tile: their four scales share a 16-byte piece of the tiled layout.  Neighbouring threads take
// neighbouring blocks, so a warp's reads (1 KB a row) and packed writes
// are contiguous.  (A thread with four neighbouring blocks of a row needs no exchange of scale bytes,
// but its 128-byte stride filled the load/store pipe: 148 instead of 131 us.)
//   packed (B, S, H, D/2), lin (B, S, H, D/16) or null, tiled (B, H, ceil(S/128), D/64, 512) or null
//
// V, blocks along the keys: a CTA transposes a tile of 128 keys x 128 d through shared memory (16-byte
// chunks swizzled by the key block, so that the row-wise fill and the column-wise reads are both
// conflict free); a thread takes two neighbouring d and one block of 16 keys.
//   packed (B, H, Dv, s_out/2), lin (B, H, Dv, s_out/16) or null,
//   tiled (B, H, ceil(Dv/128), 2 ceil(s_out/128), 512) or null
//
// Persistent: three CTAs per SM in all, dealt to the tensors in proportion to their bytes; a CTA's next item or
// tile is on its way to shared memory (cp.async, 96 KB per SM) behind the arithmetic of the current one.
//
// What bounds it: instruction issue (68 % of the slots busy, the ALU pipe 58 %), then HBM.  q, k, v of the sizes
// above, maxima and quantise pass together: 190 us with the loads of an item in registers (two CTAs of 119
// registers per SM, 175 instructions per block of 16) and one residual step per quotient; 166 us here (157).  In
// between: three CTAs with two rows in flight in registers 174 (49 KB per SM in flight are too few); cp.async of a
// thread's own two pieces, half sectors each, 210.  No gain: units of four rows one below the other (168), the
// low halves unpacked on the FMA pipe (166), hints that keep the end of the tensors in L2 (166; other sizes 2 %).
// ---------------------------------------------------------------------------------------------

// Where a Q / K work item lies: its first row (k0 = 0), or row k0 of it.
struct RowsItem {
  int s0;                       // the row
  uint32_t blk, piece;          // blocks of 16 before it in the tensor; 16-byte pieces of tiled scales before its own
};
// What a thread copies for its warp: the 64 16-byte pieces of 32 neighbouring blocks of a row are copied by
// lane as they follow in memory (a copy of its own two would take half sectors), pieces l and l + 32 by lane l.
struct RowsLoad {
  const __nv_bfloat16 *a, *b;
  int sa, sb;                   // their rows
};
__device__ __forceinline__ RowsItem rows_item_at(const QuantJob& j, uint32_t item, int k0, RowsLoad& ld) {
  RowsItem it;
  const int rest = fast_div((int)item, j.div_nb), col = (int)item - rest * j.nb;
  const int bt = rest >> 5, l = rest & 31;
  const int b = fast_div(bt, j.div_rt), rt = bt - b * j.rt;
  const int h = fast_div(col, j.div_h), c = col - h * (j.D >> 4);
  it.s0 = rt * 128 + k0 * 32 + l;
  const uint64_t src = reinterpret_cast<uint64_t>(j.x + b * j.sb + it.s0 * j.ss + h * j.sh + c * 16);
  it.blk = ((uint32_t)b * j.S + it.s0) * (uint32_t)j.nb + col;
  it.piece = ((((uint32_t)b * j.H + h) * j.rt + rt) * (uint32_t)(j.D >> 6) + (c >> 2)) * 32u + l;
  const int lane = threadIdx.x & 31;
  ld.a = reinterpret_cast<const __nv_bfloat16*>(__shfl_sync(0xffffffffu, src, lane >> 1)) + (lane & 1) * 8;
  ld.b = reinterpret_cast<const __nv_bfloat16*>(__shfl_sync(0xffffffffu, src, 16 + (lane >> 1))) + (lane & 1) * 8;
  ld.sa = __shfl_sync(0xffffffffu, it.s0, lane >> 1);
  ld.sb = __shfl_sync(0xffffffffu, it.s0, 16 + (lane >> 1));
  return it;
}
// The rows of an item on their way to shared memory as one group of asynchronous copies.  Row k of warp w: 1 KB at
// 1024 (8 k + w) of `stage`, piece p at place p ^ (p / 8 % 2) (a lane then reads its two pieces without bank conflicts).
constexpr uint32_t kRowsStage = 4 * 8 * 1024;
__device__ __forceinline__ uint32_t piece_at(uint32_t p) { return (p ^ ((p >> 3) & 1u)) * 16; }
template <int kRows>
__device__ __forceinline__ void load_rows(const QuantJob& j, const RowsLoad& ld, uint32_t stage) {
  const uint32_t dst = stage + (threadIdx.x >> 5) * 1024 + piece_at(threadIdx.x & 31);
#pragma unroll
  for (int k = 0; k < kRows; ++k) {
    if (ld.sa + 32 * k < j.S)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 8192 * k), "l"(ld.a + 32 * k * j.ss) : "memory");
    if (ld.sb + 32 * k < j.S)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 8192 * k + 512), "l"(ld.b + 32 * k * j.ss) : "memory");
  }
}
__device__ __forceinline__ void commit_copies() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// kRows = 4: the item's four rows; 1: row k0 of them (tensors too small to fill the GPU otherwise).
template <int kRows>
__device__ __forceinline__ void quantize_rows_item(const QuantJob& j, const RowsItem& it, int k0, const uint8_t* stage,
                                                   const TensorScale& ts) {
  uint32_t bytes = 0u;          // byte k: the scale of row k
#pragma unroll
  for (int k = 0; k < kRows; ++k) {
    const uint8_t* row = stage + (8 * k + (threadIdx.x >> 5)) * 1024;
    const uint4 a = *reinterpret_cast<const uint4*>(row + piece_at(2 * (threadIdx.x & 31)));
    const uint4 b = *reinterpret_cast<const uint4*>(row + piece_at(2 * (threadIdx.x & 31) + 1));
    const Words8 raw = {{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
    float v[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      v[2 * i] = __uint_as_float(raw.w[i] << 16);
      v[2 * i + 1] = __uint_as_float(raw.w[i] & 0xffff0000u);
    }
    const float bmax = absmax16(raw);
    if (it.s0 + 32 * k < j.S) {
      uint32_t lo, hi, sfb;
      quantize_block16(v, bmax, ts, lo, hi, sfb);
      bytes |= sfb << (8 * k);
      *reinterpret_cast<uint2*>(j.packed + (uint64_t)(it.blk + 32u * k * j.nb) * 8) = make_uint2(lo, hi);
    }
  }
  // Four neighbouring lanes hold the four columns of a scale word.  kRows = 4: transpose the 4 x 4
  // bytes between them, so that lane q ends up with the word of row q and all four store.
  const int q = threadIdx.x & 3;
  int row = 0;                  // (of the item: k0 stands in s0, blk and the piece's word)
  bool mine = true;
  if (kRows == 4) {
    uint32_t p = __shfl_xor_sync(0xffffffffu, bytes, 1);
    bytes = __byte_perm(bytes, p, (q & 1) ? 0x3715 : 0x6240);
    p = __shfl_xor_sync(0xffffffffu, bytes, 2);
    bytes = __byte_perm(bytes, p, (q & 2) ? 0x3276 : 0x5410);
    row = q;
  } else {
    bytes <<= 8 * q;
    bytes |= __shfl_xor_sync(0xffffffffu, bytes, 1);
    bytes |= __shfl_xor_sync(0xffffffffu, bytes, 2);
    mine = q == 0;
  }
  if (mine && j.lin != nullptr && it.s0 + 32 * row < j.S)
    *reinterpret_cast<uint32_t*>(j.lin + (it.blk & ~3u) + (uint64_t)(32u * row * j.nb)) = bytes;
  if (mine && j.tiled != nullptr)
    *reinterpret_cast<uint32_t*>(j.tiled + (uint64_t)it.piece * 16 + (row + k0) * 4) = bytes;
}

// Where a V tile lies, and this thread's eight 16-byte pieces of it (128 keys x 16 chunks of 8 d).
struct VTile {
  int hd, kb0, bh, d0;
};
__device__ __forceinline__ VTile v_tile_at(const QuantJob& j, int tile_idx) {
  VTile t;
  const int dt = (j.D + 127) / 128;
  t.hd = fast_div(tile_idx, j.div_rt);
  t.kb0 = tile_idx - t.hd * j.rt;                  // key tile inside (b, h, d tile)
  t.bh = t.hd / dt;
  t.d0 = (t.hd - t.bh * dt) * 128;
  return t;
}
// Copies the tile into shared memory asynchronously (zeros outside of the tensor) as one group of copies.
__device__ __forceinline__ void load_v_tile(const QuantJob& j, const VTile& t, uint32_t tile) {
  const int b = fast_div(t.bh, j.div_h), h = t.bh - b * j.H;
  const __nv_bfloat16* src = j.x + b * j.sb + h * j.sh + t.d0;
  const int ch = threadIdx.x & 15;
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    const int row = (threadIdx.x >> 4) + 16 * n, key = t.kb0 * 128 + row;
    const bool in = key < j.S && t.d0 + ch * 8 < j.D;
    // (row >> 4 == n)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(tile + row * 256 + ((ch ^ n) << 4)),
                 "l"(in ? src + (int64_t)key * j.ss + ch * 8 : j.x), "r"(in ? 16 : 0)
                 : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void quantize_v_tile(const QuantJob& j, const VTile& t, const TensorScale& ts, const uint8_t* tile) {
  const int kt = j.rt, Sk = j.s_out, Dv = j.D, d0 = t.d0, k0 = t.kb0 * 128, tid = threadIdx.x;
  const int n_kb_total = Sk / 16;
#pragma unroll 1
  for (int item = tid; item < 64 * 8; item += 256) {
    const int kb = item & 7, dp = item >> 3;  // key block inside the tile, d pair
    const int d = d0 + 2 * dp;
    if (d0 + 2 * (dp & ~3) >= Dv && j.tiled == nullptr) continue;   // (whole groups of lanes: shuffles below)
    const int ch = dp >> 2, within = (dp & 3) * 4;  // chunk and byte offset of the d pair
    float v0[16], v1[16];
    uint32_t m2 = 0u;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const uint32_t w = *reinterpret_cast<const uint32_t*>(tile + (16 * kb + i) * 256 + ((ch ^ kb) << 4) + within);
      v0[i] = __uint_as_float(w << 16);
      v1[i] = __uint_as_float(w & 0xffff0000u);
      m2 = absmax2(m2, w);
    }
    uint32_t lo0, hi0, sf0, lo1, hi1, sf1;
    quantize_block16(v0, fabsf(__uint_as_float(m2 << 16)), ts, lo0, hi0, sf0);
    quantize_block16(v1, fabsf(__uint_as_float(m2 & 0xffff0000u)), ts, lo1, hi1, sf1);
    const bool key_ok = k0 + 16 * kb < Sk;
    const int64_t row0 = (int64_t)t.bh * Dv + d;
    if (key_ok && d < Dv)
      *reinterpret_cast<uint2*>(j.packed + row0 * (Sk / 2) + (k0 + 16 * kb) / 2) = make_uint2(lo0, hi0);
    if (key_ok && d + 1 < Dv)
      *reinterpret_cast<uint2*>(j.packed + (row0 + 1) * (Sk / 2) + (k0 + 16 * kb) / 2) = make_uint2(lo1, hi1);
    // scale bytes: lanes kb = 4 q .. 4 q + 3 hold one word of either layout
    if (!key_ok) sf0 = sf1 = 0;
    uint32_t w0 = sf0 << (8 * (kb & 3)), w1 = sf1 << (8 * (kb & 3));
    w0 |= __shfl_xor_sync(0xffffffffu, w0, 1);
    w0 |= __shfl_xor_sync(0xffffffffu, w0, 2);
    w1 |= __shfl_xor_sync(0xffffffffu, w1, 1);
    w1 |= __shfl_xor_sync(0xffffffffu, w1, 2);
    if ((kb & 3) == 0) {
      const int kb_global = k0 / 16 + kb;
      if (j.lin != nullptr && kb_global < n_kb_total) {
        // a word may run past the row's end when Sk/16 is not a multiple of 4: byte stores there
        uint8_t* p0 = j.lin + row0 * n_kb_total + kb_global;
        const int nvalid = n_kb_total - kb_global < 4 ? n_kb_total - kb_global : 4;
        if (nvalid == 4 && (n_kb_total & 3) == 0) {
          if (d < Dv) *reinterpret_cast<uint32_t*>(p0) = w0;
          if (d + 1 < Dv) *reinterpret_cast<uint32_t*>(p0 + n_kb_total) = w1;
        } else {
          for (int q = 0; q < nvalid; ++q) {
            if (d < Dv) p0[q] = (uint8_t)(w0 >> (8 * q));
            if (d + 1 < Dv) p0[n_kb_total + q] = (uint8_t)(w1 >> (8 * q));
          }
        }
      }
      if (j.tiled != nullptr) {
        // d rows past Dv inside the 128-row tile get their zero padding here as well
        const int64_t chunk = (int64_t)t.hd * (2 * kt) + 2 * t.kb0 + kb / 4;
        const int r0 = 2 * dp, r1 = 2 * dp + 1;
        uint8_t* base = j.tiled + chunk * 512;
        *reinterpret_cast<uint32_t*>(base + (r0 % 32) * 16 + (r0 / 32) * 4) = d < Dv ? w0 : 0u;
        *reinterpret_cast<uint32_t*>(base + (r1 % 32) * 16 + (r1 / 32) * 4) = d + 1 < Dv ? w1 : 0u;
      }
    }
  }
}

constexpr int kQuantizeCtas = 3;     // per SM
constexpr uint32_t kQuantizeSmem = 2 * 128 * 256;   // two V tiles, or two items of every thread
static_assert(kQuantizeSmem == 2 * kRowsStage, "two stages");
constexpr int kQuantizeVWeight = 28; // cost of a byte of V, that of Q and K being 16
__global__ void __launch_bounds__(256, kQuantizeCtas)
quantize_kernel(const __grid_constant__ QuantJobs jobs) {
  extern __shared__ __align__(16) uint8_t tiles[];    // V: two of [key][16 chunks of 16 B], chunk ^ (key/16)
  __shared__ float warp_max[8];
  int ji = 0;
  while (ji + 1 < jobs.n && (int)blockIdx.x >= jobs.job[ji + 1].block0) ++ji;
  const QuantJob& j = jobs.job[ji];
  const int lane = threadIdx.x & 31;
  pdl_wait();
  // the first loads of the tensor go out before the partial maxima are read: one latency, not two
  const int first = blockIdx.x - j.block0, per_round = j.blocks * 256;
  const int quarter = (int)(j.items >> 2);
  // Q / K: the CTA's item of the round (below zero: past the front of the tensor); V: its tile
  int t = (int)j.items - (j.is_v ? first + 1 : 256 * (first + 1) - (int)threadIdx.x);
  int k0 = 0;
  VTile vt;
  RowsItem it;
  const uint32_t smem = smem_u32(tiles);
  RowsLoad ld;
  RowsItem next;
  int tn = -1;
  if (j.is_v) {
    vt = v_tile_at(j, t);
    load_v_tile(j, vt, smem);
  } else if (t >= 0) {
    if (j.single) {
      k0 = t / quarter;
      it = rows_item_at(j, t - k0 * quarter, k0, ld);
      load_rows<1>(j, ld, smem);
      commit_copies();
    } else {
      it = rows_item_at(j, t, 0, ld);
      load_rows<4>(j, ld, smem);
      commit_copies();
      tn = t - per_round;
      if (tn >= 0) {
        next = rows_item_at(j, tn, 0, ld);
        load_rows<4>(j, ld, smem + kRowsStage);
      }
      commit_copies();
    }
  }
  float m = 0.f;
  for (int i = threadIdx.x; i < j.num_parts; i += 256) m = fmaxf(m, j.parts[i]);
  if (j.num_parts > 1) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) warp_max[threadIdx.x >> 5] = m;
    __syncthreads();
    m = warp_max[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) m = fmaxf(m, warp_max[w]);
  } else {
    m = j.parts[0];
  }
  const TensorScale ts = make_tensor_scale(m);
  if (j.scale_out != nullptr && first == 0 && threadIdx.x == 0) *j.scale_out = ts.g;
  if (j.is_v) {
#pragma unroll 1
    for (uint32_t buf = 0;; buf ^= 128 * 256) {
      tn = t - j.blocks;
      VTile vn = vt;
      if (tn >= 0) {
        vn = v_tile_at(j, tn);
        load_v_tile(j, vn, smem + (buf ^ (128 * 256)));
        asm volatile("cp.async.wait_group 1;" ::: "memory");
      } else {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
      __syncthreads();
      quantize_v_tile(j, vt, ts, tiles + buf);
      if (tn < 0) break;
      __syncthreads();            // the buffer is read out
      vt = vn;
      t = tn;
    }
  } else if (t >= 0) {            // (items come in whole warps; lanes ascend with the blocks)
    if (j.single) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncwarp();
      quantize_rows_item<1>(j, it, k0, tiles, ts);
    } else {
#pragma unroll 1
      for (uint32_t buf = 0;; buf ^= kRowsStage) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        quantize_rows_item<4>(j, it, 0, tiles + buf, ts);
        __syncwarp();             // (the stage is read out)
        if (tn < 0) break;
        it = next;
        tn -= per_round;
        if (tn >= 0) {
          next = rows_item_at(j, tn, 0, ld);
          load_rows<4>(j, ld, smem + buf);
        }
        commit_copies();
      }
    }
  }
}

}  // namespace fa4
