// Decode / append kernel: a handful of query rows against a long key range (head dim 128).
//
// The prefill kernels put QUERY rows on the 128 lanes of the tensor-core tile; with one query
// token per sequence 127 of them are padding and the per-block latency chain (about 3000 clocks,
// two blocks in flight) sets the pace: 0.7 TB/s of K/V.  Here the products are transposed, as
// decode kernels usually do: the 128 KEYS of a block sit on the lanes and the query rows -- the
// Sq x (query heads per kv head) rows that share this kv head, at most 32 -- on the N side
// (N = 16, or 32 for more than 16 rows):
//
//   S^T (128 keys x N rows)  = K (A operand, the tile as it is loaded) . Q^T (B operand)
//   O^T (128 dv   x N rows) += V^T (A operand: V is stored key-contiguous, i.e. already as the
//                                   K-major (dv, keys) matrix) . P^T (B operand)
//
// so no lane is wasted, an S^T buffer is N tensor-memory columns, and tensor memory hands a
// softmax thread ONE key with its <= N scores.  The warp transposes that within groups of `rows`
// lanes, after which a thread owns one query ROW with `rows` neighbouring keys: the per-row work
// (mask limit, reference maximum, block exponent, running sum) is scalar per thread; block and
// warp maxima take zero to three shuffles, the CTA maximum one exchange through shared memory per
// block.  P is quantised exactly as in the prefill kernels (e2m1, power-of-two ue4m3 scale per
// row and 16 keys, lazy reference).
//
// One CTA = one (split, kv head, batch entry): a contiguous share of the entry's 128-key blocks,
// visited in ascending order; its normalised fp32 partial O and partial LSE are merged inside the
// cluster of an entry's splits (up to eight), or by combine_splits_kernel as on the split-KV path of
// attn_ws.cuh.  Grid = (splits, Hkv, B).  Batches whose entries have key counts in memory and many keys are dealt to the
// CTAs by those counts instead, where the caller leaves the splits open (kBalanced): equal splits leave a batch of lengths spread over the logarithm waiting
// for the longest entry's CTAs with four fifths of the GPU idle.  us, 16 entries up to 8192 keys, 8 heads, GQA 4 18.5 ->
// 14.4, four tokens 34.1 -> 17.7; 32 up to 16384 57.3 -> 33.2 (143 MB of keys: 22 us at the copy bandwidth); 5 up to
// 51200, 32 heads 131 -> 65.
//   warps 0-3  softmax / correction / epilogue (thread = key lane, after the transpose a row; in the
//              correction and the epilogue a dv lane)
//   warps 8-11 up to eight rows: a second softmax warpgroup, which takes the odd blocks; in the deep form
//              warps 8-19: three more, the blocks dealt in turn
//   warp 4     TMA producer of K (ring of three tiles, through the page table if there is one)
//   warp 5     issuer of K . Q^T (owns tensor memory)
//   warp 6     TMA producer of V (its own ring, independent of K's)
//   warp 7     issuer of V^T . P^T
// Every wait is bounded, like everywhere else.
//
// Most calls are over in 6-20 us, and whatever runs once per CTA -- set-up, epilogue, merge -- runs from cold
// instruction memory: its length in code, not in work, is its time.  So what is the same for all lanes of a row is
// done by the lanes of that row at once instead of row after row in unrolled code, divisions are multiplications, and
// the merge takes a row a warp.  us, code unrolled over the rows -> this: 32 rows (GQA 4, eight tokens), 2 entries of up
// to 16384 keys 42.2 -> 26.2; 16 rows, 4 x 8192 21.6 -> 18.0; 4 rows, paged batch of 16 up to 8192 20.7 -> 18.7 (with
// combine_splits_kernel written the same way 21.9, 16.6, 18.7).
#pragma once
#include "attn_common.cuh"
#include "softmax.cuh"

namespace fa4 {
namespace dec {

// K and V tiles, S^T buffers (N columns each) and P^T tiles (N rows x 64 bytes) with their scale chunks:
// kDepth of each.  Three let THREE CTAs share an SM (70 KB of shared memory, 128 tensor-memory columns),
// five let two (115 KB, 256 columns).  A CTA's loads are bound by their latency, kDepth x 18 KB per round
// trip, so five are better whenever no third CTA is there to run.
// (Registers: three CTAs of 384 threads leave 56, two of 640 leave 48, and up to eight rows the kernel wants more.  Bytes
// of spill stores, merging / not: shallow 4 / 28, with linear scales 96 / 112-136; deep, four rows 48 / 84, 176 / 100;
// eight rows 100 / 40, 212 / 136.  None above eight rows.  Balanced, shallow: 16-24, with linear scales 76-132.  With them the deep form is still the faster one for
// ragged batches, see softmax_wgs, and reading linear scales faster than a launch of its own, see linear_keys_limit in
// host.cpp, whose line is nearer for five to eight rows.)
constexpr int kMaxCluster = 8;  // splits that are merged inside a cluster (portable cluster size)
constexpr int kMaxRows = 32; // query rows per kv head: Sq * group
// Limits of a balanced call (see balance(), which counts in floats): entries; keys of one, blocks of all, CTAs.
constexpr int kMaxBalanced = 128, kMaxBalancedKeys = 1 << 26, kMaxBalancedBlocks = (1 << 20) - 8192, kMaxBalancedCtas = 4095;
// Blocks below which a unit is not cut further.  (Two, three, four: one token, 48 entries up to 4096 keys of one head 10.7,
// 10.6, 10.7 us; four tokens, 6 entries up to 2048 of 8 heads 9.6, 9.8, 11.0.)
constexpr int kMinBlocks = 3;
// log2 units by which references may fall, in all, below the highest one that a row has had in its CTA: O and the row sum
// grow by as much (2^64 on top of the 2^10 of a weight, the 2^12 of a value and the 2^26 of the keys), and what lies further down
// is nothing beside what is there.
constexpr float kMaxFall = 64.f;
// Softmax warpgroups: one above eight rows; up to eight, two in the shallow form (registers: three CTAs of
// twelve warps per SM leave 56 per thread) and four in the deep one, whose long entries run on with few CTAs
// beside them: a block is a chain of some 1700 clocks in its warpgroup, and only the reference is handed
// from block to block.  Blocks are dealt in turn.  us, two warpgroups -> four: 32 paged sequences up to 16384
// 66.6 -> 61.0, 16 up to 8192 20.25 -> 20.23 (there the loads of a CTA pace it).
__host__ __device__ constexpr int softmax_wgs(int rows, int depth) {
  return rows > 8 ? 1 : (depth == 5 ? 4 : 2);
}
__host__ __device__ constexpr int strands_of(int rows) { return rows <= 8 ? 4 : 1; }
__host__ __device__ constexpr int threads_of(int rows, int depth) { return 128 + 128 * softmax_wgs(rows, depth); }

// shared memory of the form with kN rows per operand and kWgs softmax warpgroups
template <int kDepth, int kN, int kWgs>
struct Smem {
  static constexpr uint32_t kQBytes = kN * 64;                      // Q^T / P^T operand: rows of 64 bytes
  static constexpr uint32_t kOffK = 0;
  static constexpr uint32_t kOffV = kOffK + kDepth * kTileBytes;
  static constexpr uint32_t kOffSFK = kOffV + kDepth * kTileBytes;
  static constexpr uint32_t kOffSFV = kOffSFK + kDepth * kSfBytes;
  static constexpr uint32_t kOffQ = kOffSFV + kDepth * kSfBytes;    // rows x 64 bytes, 64-byte swizzle
  static constexpr uint32_t kOffSFQ = kOffQ + kQBytes;              // two 512-byte chunks
  static constexpr uint32_t kOffP = kOffSFQ + 1024;                 // kDepth x kQBytes
  static constexpr uint32_t kOffSFP = kOffP + kDepth * kQBytes;     // kDepth x 2 chunks x 512
  static constexpr uint32_t kOffRed = kOffSFP + kDepth * 1024;      // WGs x 2 x 4 warps x kN floats
  static constexpr uint32_t kOffHand = kOffRed + kWgs * 2 * 4 * kN * 4;   // WGs x 4 warps x kN references
  static constexpr uint32_t kOffSum = kOffHand + kWgs * 4 * kN * 4;       // kWgs = 2: 2 x 256 (row sum, its reference)
  static constexpr uint32_t kOffOld = kOffSum + (kWgs == 2 ? 2 * 256 * 8 : 0);   // kWgs = 2: WGs x (4 warps' sums, 1 reference) x kN
  static constexpr uint32_t kOffBar = kOffOld + (kWgs == 2 ? kWgs * 5 * kN * 4 : 0);
  // barriers
  static constexpr uint32_t kKFull = 0, kVFull = kKFull + kDepth, kSFull = kVFull + kDepth, kSFree = kSFull + kDepth,
                            kPFull = kSFree + kDepth, kPvDone = kPFull + kDepth, kQReady = kPvDone + kDepth,
                            kSync = kQReady + 1 /* WGs */, kHand = kSync + kWgs /* WGs x 4 */, kFin = kHand + 4 * kWgs,
                            kDrain = kFin + 1 /* 2 */, kCount = kDrain + 2;
  static constexpr uint32_t kOffMisc = (kOffBar + 8 * kCount + 15) / 16 * 16;
  static constexpr uint32_t kOffWork = (kOffMisc + 16 + sizeof(WaitCtx) + 15) / 16 * 16;   // DecodeWork
  static constexpr uint32_t kRequest = kOffWork + 48 + 1024;
  // (1 KB per CTA is the system's)
  static_assert((kDepth == 3 ? 3 : 2) * (kRequest + 1024) <= 228 * 1024, "decode kernel shared memory");
};

template <int kRows, int kDepth>
using form = Smem<kDepth, (kRows <= 16 ? 16 : 32), softmax_wgs(kRows, kDepth)>;   // of the kernel's form

// tensor memory of the form with N columns per operand: S^T buffers, O^T, scale factors.  The K / V / P
// scale slots alternate between two copies: the copy and the product that reads it are issued by one
// thread to the in-order tensor pipe, the second copy keeps a copy from racing the product before.
template <int kN, int kDepth>
struct Tm {
  static constexpr uint32_t kCols = kDepth == 3 ? 128 : 256;
  static constexpr uint32_t kS = 0 /* kDepth x N */, kO = kDepth * kN, kSFQ = kO + kN, kSFK = kSFQ + 8 /* 2 x 8 */,
                            kSFV = kSFK + 16 /* 2 x 8 */, kSFP = kSFV + 16 /* 2 x 8 */;
  static_assert(kSFP + 16 <= kCols, "tensor-memory map of the decode kernel");
};

enum Site { kDKFull = 80, kDVFull, kDKFree, kDVFree, kDSFull, kDSFree, kDPFull, kDPvDone, kDQReady, kDSync, kDHand, kDFin };

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
      ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
      "r"(r[15]), "r"(taddr)
      : "memory");
}

// One e2m1 byte from two values: `lo` goes to the low nibble (the even key).
__device__ __forceinline__ uint32_t pack2_e2m1(float lo, float hi) {
  uint16_t b;
  asm("{\n"
      ".reg .b8 t;\n"
      "cvt.rn.satfinite.e2m1x2.f32 t, %2, %1;\n"
      "cvt.u16.u8 %0, t;\n"
      "}\n"
      : "=h"(b)
      : "f"(lo), "f"(hi));
  return b;
}

// kN columns (4, 8 or 16) of this thread's tensor-memory lane.
template <int kN>
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t* r) {
  if constexpr (kN == 4) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr)
                 : "memory");
  } else if constexpr (kN == 8) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
  } else if constexpr (kN == 16) {
    tmem_ld16(taddr, r);
  } else {
    tmem_ld32(taddr, r);
  }
}
template <int kN>
__device__ __forceinline__ void tmem_st_cols(uint32_t taddr, const uint32_t* r) {
  if constexpr (kN == 4) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%4], {%0, %1, %2, %3};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(taddr)
                 : "memory");
  } else if constexpr (kN == 8) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                 "r"(taddr)
                 : "memory");
  } else if constexpr (kN == 16) {
    tmem_st16(taddr, r);
  } else {
    tmem_st32(taddr, r);
  }
}

// T x T transpose inside every group of T neighbouring lanes (T = 4, 8, 16, 32): before, lane i of a
// group holds x[0..T) = its own column; after, x[j] is what lane j of the group held in x[i].
// log2(T) butterfly rounds of T / 2 shuffles.
template <int T>
__device__ __forceinline__ void lane_group_transpose(float (&x)[T], int lane) {
#pragma unroll
  for (int bit = 1; bit < T; bit <<= 1) {
    const bool up = (lane & bit) != 0;
#pragma unroll
    for (int j = 0; j < T; ++j) {
      if ((j & bit) == 0) {
        const float send = up ? x[j] : x[j | bit];
        const float recv = __shfl_xor_sync(0xffffffffu, send, bit);
        if (up) x[j] = recv; else x[j | bit] = recv;
      }
    }
  }
}

// Exponent of one 16-key block of P from its maximum (the scalar form of block_exponents4):
// noff with p'/2^e = 2^(s * sl2 + noff), and the byte e + 127.
__device__ __forceinline__ void block_exponent1(float bm, float m_ref, float sl2, float& noff,
                                                uint32_t& ue) {
  constexpr float kMagic = 12582912.f + 127.f;
  const float msc = (m_ref == kNegInf) ? 0.f : __fmul_rn(m_ref, sl2);   // (not contracted: one result in all forms)
  const float c_t = static_cast<float>(kShift) - kLog2Of6 + 0.4999995f - msc;
  const float c_off = static_cast<float>(kShift) - msc;
  float t = fmaf(bm, sl2, c_t);
  t = fmaxf(t, static_cast<float>(kEMin) - 0.4f);
  const float u = t + kMagic;
  ue = __float_as_uint(u) & 0xffu;
  noff = c_off - (u - kMagic);
}

}  // namespace dec

// Linear scale factors as a caller's cache holds them: q (B, Sq, Hq, 8), k (B, Sk, Hkv, 8), v (B, Hkv, 128, columns)
// bytes, any strides in the outer dimensions and any alignment.
struct LinearScales {
  const uint8_t *q, *k, *v;
  int64_t q_b, q_s, q_h, k_b, k_s, k_h, v_b, v_h, v_d;
  int k_rows, v_cols;    // rows of k and columns of v of an entry (of a page)
};

// How the CTAs of the balanced form are dealt, see balance().  Its partials: ctas x (Sq * group) x 128 floats in
// o_partial, as many LSEs in lse_partial.
struct Balance {
  int ctas, slots;       // of the grid; at once on the GPU
  int min_per, rounds;
  float inv_slots, inv_extra;   // 1 / slots, 1 / (ctas - B * Hkv)
  int2* pieces;          // (B, Hkv): first CTA and number of CTAs
};

struct DecodeParams {
  const uint8_t* q;      // (B, Sq, Hq, 64) packed e2m1
  const uint8_t* q_sf;   // tiled (B, Hq, ceil(Sq/128), 2, 512)
  int64_t q_stride_b, q_stride_s, q_stride_h;
  int num_splits;
  float* o_partial;      // (splits, B, Sq, Hq, 128) fp32
  float* lse_partial;    // (splits, B, Hq, Sq) fp32
  LinearScales lin;      // kLinear
  Balance balance;       // kBalanced
};

// How the splits of a (kv head, batch entry) become one result.
enum DecodeMerge {
  kWorkspace,   // partials to o_partial / lse_partial, merged by combine_splits_kernel
  kCluster,     // the splits are one cluster, which merges them through distributed shared memory
  kBalanced     // entries of unequal lengths, CTAs dealt by the lengths: see balance()
};

// What a CTA of the balanced form works on: blocks i0 .. i0 + n - 1 of kv head hk of entry b, the `piece`-th of `pieces`.
struct alignas(16) DecodeWork {
  int b, hk, piece, pieces;   // b < 0: nothing
  int i0, n, share, into;     // share: blocks of a split; into: those of i0's split before i0
  int sk, pad[3];             // keys of the entry
};

// Whole quotient of numbers below 2^20 (the exact one is off the next integer by more than the reciprocal's error).
__device__ __forceinline__ int small_div(int n, float inv) { return (int)(((float)n + 0.5f) * inv); }
static_assert(sizeof(DecodeWork) == 48, "its place in shared memory");
// Entries of unequal lengths (key counts in memory): the grid is dealt by the lengths.  A unit (kv head, entry) is cut
// into the fewest pieces of at most `per` blocks, and `per` is the smallest number, from the mean of a resident CTA on,
// for which the grid has the CTAs.  With more CTAs than fit at once (d.balance.rounds > 1) entries come by length, the
// longest first, to within a factor of two.  Run by one warp; `len`: B words of shared memory.
__device__ __forceinline__ DecodeWork balance(const KernelParams& p, const DecodeParams& d, int lane, int* len) {
  const int cid = blockIdx.x;
  int longest = 0, total = 0;
#pragma unroll 1
  for (int e = lane; e < p.B; e += 32) {
    const int used = p.seqused_k[e];
    const int sk = used < 0 ? 0 : (used < p.Sk ? used : p.Sk);
    const int n = (sk + kBlockN - 1) / kBlockN;
    len[e] = sk;
    longest = max(longest, n);
    total += n;
  }
  longest = __reduce_max_sync(0xffffffffu, longest);
  total = __reduce_add_sync(0xffffffffu, total) * p.Hkv;
  __syncwarp();
  auto pieces_of = [&](int e, int per, float inv) -> int {
    return max(1, small_div((len[e] + kBlockN - 1) / kBlockN + per - 1, inv));
  };
  // (as many pieces as units, and what the whole list has of `hi`: always enough)
  int lo = max(d.balance.min_per, small_div(total + d.balance.slots - 1, d.balance.inv_slots));
  int hi = max(lo, min(longest, small_div(total, d.balance.inv_extra) + 1));
#pragma unroll 1
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    const float inv = __frcp_rn((float)mid);
    int c = 0;
#pragma unroll 1
    for (int e = lane; e < p.B; e += 32) c += pieces_of(e, mid, inv);
    if (__reduce_add_sync(0xffffffffu, c) * p.Hkv <= d.balance.ctas) hi = mid; else lo = mid + 1;
  }
  const float inv = __frcp_rn((float)lo);
  DecodeWork w;
  w.b = -1; w.hk = 0; w.piece = 0; w.pieces = 1; w.i0 = 0; w.n = 0; w.share = 1; w.into = 0; w.sk = 0;
  int at = cid;           // less the CTAs of the entries passed so far
#pragma unroll 1
  for (int round = 0; round < d.balance.rounds && w.b < 0; ++round) {
    const int top = longest >> round, bottom = round + 1 < d.balance.rounds ? top >> 1 : -1;
#pragma unroll 1
    for (int e0 = 0; e0 < p.B; e0 += 32) {
      int mine = 0;
      if (e0 + lane < p.B) {
        const int n = (len[e0 + lane] + kBlockN - 1) / kBlockN;
        if (n <= top && n > bottom) mine = max(1, small_div(n + lo - 1, inv));
      }
      int upto = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
      }
      const uint32_t hit = __ballot_sync(0xffffffffu, at < upto * p.Hkv);
      if (hit != 0u) {
        const int l = __ffs(hit) - 1;
        w.b = e0 + l;
        w.pieces = __shfl_sync(0xffffffffu, mine, l);
        at -= (__shfl_sync(0xffffffffu, upto, l) - w.pieces) * p.Hkv;
        break;
      }
      at -= __shfl_sync(0xffffffffu, upto, 31) * p.Hkv;
    }
  }
  if (w.b >= 0) {
    const float inv_pieces = __frcp_rn((float)w.pieces);
    w.hk = small_div(at, inv_pieces);
    w.piece = at - w.hk * w.pieces;
    w.sk = len[w.b];
    const int n = (w.sk + kBlockN - 1) / kBlockN, each = small_div(n + w.pieces - 1, inv_pieces);
    w.share = max(1, fast_div(n + d.num_splits - 1, p.div_splits));
    w.i0 = min(n, w.piece * each);
    w.n = min(n - w.i0, each);
    w.into = w.i0 - w.share * small_div(w.i0, __frcp_rn((float)w.share));
    if (lane == 0 && w.piece == 0) d.balance.pieces[w.b * p.Hkv + w.hk] = make_int2(cid, w.pieces);
  }
  return w;
}

// kR: query rows the softmax code is built for (4, 8, 16 or 32 >= Sq * group): the size of the
// lane-group transpose and the number of keys a thread owns afterwards.  N (the MMA's N, the
// columns of an S^T buffer) is 16 up to sixteen rows and 32 above.
// kMerge: the splits of a (kv head, batch entry) are one cluster, which merges their partials through
// distributed shared memory and writes the result; otherwise they go to o_partial / lse_partial.
// kLinear: the scales come in the caller's linear layouts, and the producers put them into tiles on the way: a lane
// reads the eight bytes of four rows, two blocks at a time and ahead of the ones it stores.  For short calls, of which
// the launch that tiles the scales is a third; with many keys the reads, a 32-byte sector for eight bytes,
// take longer than that launch (the line lies in host.cpp).
template <int kR, DecodeMerge kHow, int kDepth, bool kLinear>
__global__ void __launch_bounds__(dec::threads_of(kR, kDepth), kDepth == 3 ? 3 : 2)
attn_decode_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                   const KernelParams p, const DecodeParams d) {
  using namespace dec;
  constexpr bool kBal = kHow == kBalanced, kMerge = kHow == kCluster;
  constexpr int kWgs = softmax_wgs(kR, kDepth);
  constexpr int kN = kR <= 16 ? 16 : 32, kMaxRows = kN;   // (stride of the arrays per row)
  using L = form<kR, kDepth>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gbase = smem_raw + (base - smem_u32(smem_raw));
  auto bar = [&](uint32_t idx) -> uint32_t { return base + L::kOffBar + 8u * idx; };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gbase + L::kOffMisc);
  volatile uint32_t* s_abort = reinterpret_cast<volatile uint32_t*>(gbase + L::kOffMisc + 4);
  volatile float* s_red = reinterpret_cast<volatile float*>(gbase + L::kOffRed);    // [WGs][2][4][rows]
  volatile float* s_old = reinterpret_cast<volatile float*>(gbase + L::kOffOld);
  volatile float* s_hand = reinterpret_cast<volatile float*>(gbase + L::kOffHand);  // [WGs][4][rows]
  using TM = Tm<kN, kDepth>;
  constexpr int kStrands = strands_of(kR), kOwn = kStrands / kWgs;   // partial row sums; of a warpgroup

  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int split = kBal ? 0 : blockIdx.x;
  int hk = blockIdx.y, b = blockIdx.z;
  WaitCtx& wc = *reinterpret_cast<WaitCtx*>(gbase + L::kOffMisc + 16);
  const int R = p.Sq * p.group;  // live query rows (<= kR)

  if (tid == 0) {
    *s_abort = 0u;
    wc = WaitCtx{s_abort, p.status, p.budget_ns, p.epoch};
    for (int s = 0; s < kDepth; ++s) {
      mbar_init(bar(L::kKFull + s), 1);
      mbar_init(bar(L::kVFull + s), 1);
      mbar_init(bar(L::kSFull + s), 1);
      mbar_init(bar(L::kSFree + s), 128);
      mbar_init(bar(L::kPFull + s), 128);
      mbar_init(bar(L::kPvDone + s), 1);
    }
    mbar_init(bar(L::kQReady), 128);
    for (int w = 0; w < kWgs; ++w) mbar_init(bar(L::kSync + w), 128);
    for (int w = 0; w < 4 * kWgs; ++w) mbar_init(bar(L::kHand + w), 32);
    mbar_init(bar(L::kFin), 128 * (kWgs > 1 ? kWgs - 1 : 1));
    for (int w = 0; w < 2; ++w) mbar_init(bar(L::kDrain + w), 1);
    fence_barrier_init();
  }
  if (warp == 4 && lane == 0) tma_prefetch_desc(&tm_k);
  if (warp == 6 && lane == 0) tma_prefetch_desc(&tm_v);
  if (warp == 5) {
    tmem_alloc(base + L::kOffMisc, TM::kCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  pdl_wait();
  DecodeWork work;
  if constexpr (kBal) {
    // (the memory of the softmax warps' exchanges is free until the first scores)
    static_assert(L::kOffBar - L::kOffRed >= 4 * kMaxBalanced, "scratch");
    DecodeWork* slot = reinterpret_cast<DecodeWork*>(gbase + L::kOffWork);
    if (warp == 0) {
      const DecodeWork w = balance(p, d, lane, reinterpret_cast<int*>(gbase + L::kOffRed));
      if (lane == 0) *slot = w;
    }
    __syncthreads();
    work = *slot;
    tc_fence_after_sync();
    if (work.b < 0) {
      if (warp == 5) tmem_dealloc(*tmem_slot, TM::kCols);
      return;
    }
    hk = work.hk;
    b = work.b;
  }
  // The query rows and their scale words go to registers before anything else is read: their
  // latency (a trip to HBM while every CTA of the grid starts its K / V stream) then overlaps the
  // rendezvous below.  Threads 0-127: row tid / 4, 16-byte chunk tid % 4; threads 0-63
  // also: row tid / 2, the scale word of 64-element step tid % 2.
  uint4 q_pref = make_uint4(0u, 0u, 0u, 0u);
  uint32_t qsf_pref = 0u;
  if (tid < 128) {
    const int r = tid >> 2, ch = tid & 3;
    if (r < R) {
      const int s = fast_div(r, p.div_group), h = hk * p.group + r - s * p.group;
      q_pref = *reinterpret_cast<const uint4*>(d.q + b * d.q_stride_b + s * d.q_stride_s + h * d.q_stride_h +
                                               ch * 16);
    }
  }
  if (tid < 64) {
    const int r = tid >> 1, ks = tid & 1;
    if (r < R) {
      const int s = fast_div(r, p.div_group), h = hk * p.group + r - s * p.group;
      if constexpr (kLinear) {
        const uint8_t* src = d.lin.q + b * d.lin.q_b + s * d.lin.q_s + h * d.lin.q_h + 4 * ks;
        qsf_pref = src[0] | (uint32_t)src[1] << 8 | (uint32_t)src[2] << 16 | (uint32_t)src[3] << 24;
      } else {
        const uint8_t* chunk = d.q_sf + b * p.qsf_stride_b + h * p.qsf_stride_h + ((int64_t)(s / 128) * 2 + ks) * 512;
        const int rr = s % 128;
        qsf_pref = *reinterpret_cast<const uint32_t*>(chunk + (rr % 32) * 16 + (rr / 32) * 4);
      }
    }
  }

  // this CTA's share of the entry's K/V blocks (ascending, contiguous, ceil division like the
  // split-KV path of the prefill kernel)
  int sk = p.Sk;
  if constexpr (kBal) {
    sk = work.sk;
  } else if (p.seqused_k != nullptr) {
    const int used = p.seqused_k[b];
    sk = used < 0 ? 0 : (used < p.Sk ? used : p.Sk);
  }
  int i0, n;
  // kBalanced: the references of the rows follow the splits, not the CTAs: a reference starts anew with every split (at
  // li = next_start), and a CTA that begins inside of one visits that one's first block before its own (pre = 1), for the
  // reference alone.  (It is worked on like the others, with weights of zero.  Without its V tile, P and product: the same bits, and no
  // faster: 16 entries up to 8192 keys, lengths spread 13.6 -> 13.8 us, a tenth 11.1 -> 11.1.)  P is then rounded as with a CTA per split, but for rows whose
  // reference moves inside of a split, in blocks that the CTA passes over.
  int pre = 0, next_start = 1 << 30;
  if constexpr (kBal) {
    pre = work.n > 0 && work.into > 0 ? 1 : 0;
    i0 = work.i0 - pre;
    n = work.n + pre;
    next_start = pre + work.share - work.into;
  } else {
    const int n_total = (sk + kBlockN - 1) / kBlockN;
    const int per = fast_div(n_total + d.num_splits - 1, p.div_splits);
    i0 = split * per < n_total ? split * per : n_total;
    n = (i0 + per < n_total ? i0 + per : n_total) - i0;
  }
  // (producers) lane l: where the CTA's block li + l lies: batch coordinate, block inside it
  auto locate = [&](int li) -> int2 {
    int2 r = make_int2(b, i0 + li + lane);
    if (kBal && pre != 0 && li + lane == 0) r.y = work.i0 - work.into;
    if (p.page_table != nullptr && li + lane < n) {
      const int pg = fast_div(r.y, p.div_page);
      r.x = p.page_table[(int64_t)b * p.pages_per_seq + pg];
      r.y -= pg * (p.page_size / kBlockN);
    }
    return r;
  };
  int2 at = make_int2(0, 0);
  // kLinear: the scale words of blocks fetched, fetched + 1: rows l, l + 32, l + 64, l + 96 of lane l, three aligned words
  // around the eight bytes of a row, which start `shift` bits into the first one (the same in the four rows, 32 strides
  // apart).  Words without a byte of the tensor are not read.
  uint32_t words[kLinear ? 2 : 1][4][3], shift[2] = {0u, 0u};
  auto fetch = [&](int li0) {
    if constexpr (kLinear) {
      const bool is_k = warp == 4;
      const int64_t row_stride = is_k ? d.lin.k_s : d.lin.v_d;
      const uint8_t* head = is_k ? d.lin.k + hk * d.lin.k_h : d.lin.v + hk * d.lin.v_h;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int li = li0 + u;
        const int kb = __shfl_sync(0xffffffffu, at.x, li & 31), nbl = __shfl_sync(0xffffffffu, at.y, li & 31);
        if (li < n) {
          const int left = is_k ? d.lin.k_rows - nbl * kBlockN : d.lin.v_cols - nbl * 8;   // rows, bytes of a row
          const uint8_t* src = head + kb * (is_k ? d.lin.k_b : d.lin.v_b) + (is_k ? nbl * kBlockN * row_stride : nbl * 8) +
                               lane * row_stride;
          const uint32_t skew = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 3u);
          const uint32_t end = skew + (is_k || left > 8 ? 8u : (uint32_t)left);
          shift[u] = 8u * skew;
          src -= skew;
#pragma unroll
          for (int c = 0; c < 4; ++c, src += 32 * row_stride) {
            const bool row_ok = !is_k || c * 32 + lane < left;
#pragma unroll
            for (int x = 0; x < 3; ++x)
              words[u][c][x] = row_ok && 4u * x < end ? *reinterpret_cast<const uint32_t*>(src + 4 * x) : 0u;
          }
        }
      }
    }
  };
  if (warp == 4 || warp == 6) {
    at = locate(0);
    if (kLinear) fetch(0);
  }
  if constexpr (!kBal) {
    __syncthreads();
    tc_fence_after_sync();
  }
  pdl_trigger();
  const uint32_t tmem = *tmem_slot;
  const ScoreScales sc = score_scales(p);
  constexpr uint32_t idesc = make_idesc_nvf4(128, kN);
  bool ok = true;

  if (warp == 4 || warp == 6) {
    // ============================================ TMA producers =================================
    // Warp 4 streams K, warp 6 streams V, each as far ahead as its own ring allows.  (One thread
    // issuing K and V in turn tied the K stream to the P V products: K of block i + 1 went out
    // only when P V of block i - 3 had freed a V stage, one block time before Q K^T needs it, and
    // the kernel ran at one block per memory latency.)
    // Where the blocks lie (a page of the pool and the block in it) is looked up by the whole warp, a block a
    // lane and 32 blocks at a time, the first ones before the CTA's set-up is over: read one by one in front of each
    // load, the table held the K stream to a block per latency, 700 clocks, which four softmax warpgroups outrun.
    const bool is_k = warp == 4;
    // (a K stage is free once its scores are in tensor memory, a V stage once its product is in O: no
    // commits of their own)
    const uint32_t full0 = is_k ? L::kKFull : L::kVFull, free0 = is_k ? L::kSFull : L::kPvDone;
    const uint32_t tile0 = base + (is_k ? L::kOffK : L::kOffV), sf0 = base + (is_k ? L::kOffSFK : L::kOffSFV);
    const uint8_t* sf_src = is_k ? p.k_sf + hk * p.ksf_stride_h : p.v_sf + hk * p.vsf_stride_h;
    const int64_t sf_stride_b = is_k ? p.ksf_stride_b : p.vsf_stride_b;
    auto load_tile = [&](int st, int kb, int nbl) {
      if (is_k) tma_load_4d(tile0 + st * kTileBytes, &tm_k, bar(full0 + st), 0, hk, nbl * kBlockN, kb);
      else tma_load_4d(tile0 + st * kTileBytes, &tm_v, bar(full0 + st), nbl * (kBlockN / 2), 0, hk, kb);
    };
    int li = 0;
    for (; li < n; ++li) {
      if ((li & 31) == 0 && li > 0 && !kLinear) at = locate(li);
      const uint32_t st = li % kDepth;
      const int kb = __shfl_sync(0xffffffffu, at.x, li & 31), nbl = __shfl_sync(0xffffffffu, at.y, li & 31);
      const bool lead = elect_one();
      if (lead) {
        if (li >= kDepth) ok = mbar_wait(bar(free0 + st), ((li - kDepth) / kDepth) & 1, wc, is_k ? kDKFree : kDVFree);
        if (ok) {
          if constexpr (kLinear) mbar_expect_tx(bar(full0 + st), kTileBytes);
          else mbar_arrive_expect_tx(bar(full0 + st), kTileBytes + kSfBytes);
          load_tile(st, kb, nbl);
          if constexpr (!kLinear)
            bulk_load(sf0 + st * kSfBytes, sf_src + kb * sf_stride_b + (int64_t)nbl * kSfBytes, kSfBytes, bar(full0 + st));
        }
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      if constexpr (kLinear) {
        // the stage is free (its leader waited): both chunks of the block, 16 bytes a lane; the tile's barrier
        // completes with the copy and with this arrival
        const int u = li & 1;
        const int left = is_k ? 8 : d.lin.v_cols - nbl * 8;
        uint32_t lo[4], hi[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint32_t w0 = u ? words[1][c][0] : words[0][c][0], w1 = u ? words[1][c][1] : words[0][c][1],
                         w2 = u ? words[1][c][2] : words[0][c][2], sh = u ? shift[1] : shift[0];
          lo[c] = __funnelshift_r(w0, w1, sh);
          hi[c] = __funnelshift_r(w1, w2, sh);
          if (left < 8) {                       // (bytes past the row's end are zero)
            lo[c] &= left < 4 ? (1u << (8 * left)) - 1u : 0xffffffffu;
            hi[c] &= left <= 4 ? 0u : (1u << (8 * (left - 4))) - 1u;
          }
        }
        uint8_t* dst = gbase + (is_k ? L::kOffSFK : L::kOffSFV) + st * kSfBytes + lane * 16;
        *reinterpret_cast<uint4*>(dst) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        *reinterpret_cast<uint4*>(dst + 512) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lead) mbar_arrive(bar(full0 + st));
        if (u == 1) {
          if (((li + 1) & 31) == 0) at = locate(li + 1);
          fetch(li + 1);
        }
      }
    }
    if (!ok && lane == 0) {
      // bounded drain: let the copies already issued (those of the blocks before li) land before the CTA's memory
      // is released
      const uint64_t t0 = globaltimer_ns();
      for (int i = li > kDepth ? li - kDepth : 0; i < li; ++i) {
        while (!mbar_try_wait(bar(full0 + (i % kDepth)), (i / kDepth) & 1) &&
               globaltimer_ns() - t0 < 50ull * 1000 * 1000) {}
      }
    }
  } else if (warp == 5) {
    // ============================================ K . Q^T issuer ===============================
    // (One thread that issued both products paced the kernel while an issuing thread took 100 clocks for each of a
    // block's fourteen copies, products and commits, see elect_one.  Two threads stay: the second product's waits would
    // hold up the first.)
    if (elect_one() && n > 0) {
      ok = mbar_wait(bar(L::kQReady), 0, wc, kDQReady);
      uint64_t dq[2];
      if (ok) {
        tc_fence_after_sync();
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
          tc_cp_sf(tmem + TM::kSFQ + 4 * ks, base + L::kOffSFQ + 512 * ks);
          dq[ks] = make_desc_sw64(base + L::kOffQ + 32 * ks);
        }
      }
      for (int li = 0; ok && li < n; ++li) {
        const uint32_t st = li % kDepth, buf = li % kDepth;
        ok = mbar_wait(bar(L::kKFull + st), (li / kDepth) & 1, wc, kDKFull);
        if (!ok) break;
        if (li >= kDepth) {
          ok = mbar_wait(bar(L::kSFree + buf), ((li - kDepth) / kDepth) & 1, wc, kDSFree);
          if (!ok) break;
        }
        tc_fence_after_sync();
        const uint32_t sfk = tmem + TM::kSFK + 8 * (li & 1);
        const uint32_t kt = base + L::kOffK + st * kTileBytes, ksf = base + L::kOffSFK + st * kSfBytes;
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) tc_cp_sf(sfk + 4 * ks, ksf + 512 * ks);
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
          mma_nvf4(tmem + TM::kS + kN * buf, make_desc_sw64(kt + 32 * ks), dq[ks], idesc, sfk + 4 * ks,
                   tmem + TM::kSFQ + 4 * ks, ks > 0 ? 1u : 0u);
        }
        tc_commit(bar(L::kSFull + buf));   // scores ready; also: the K stage is free
      }
      if (!ok) {
        const uint64_t t0 = globaltimer_ns();
        tc_commit(bar(L::kDrain));
        while (!mbar_try_wait(bar(L::kDrain), 0) && globaltimer_ns() - t0 < 50ull * 1000 * 1000) {}
      }
    }
  } else if (warp == 7) {
    // ============================================ V^T . P^T issuer =============================
    if (elect_one()) {
      for (int li = 0; ok && li < n; ++li) {
        const uint32_t st = li % kDepth, slot = li % kDepth;
        ok = mbar_wait(bar(L::kVFull + st), (li / kDepth) & 1, wc, kDVFull);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t sfv = tmem + TM::kSFV + 8 * (li & 1), sfp = tmem + TM::kSFP + 8 * (li & 1);
        const uint32_t vt = base + L::kOffV + st * kTileBytes, vsf = base + L::kOffSFV + st * kSfBytes;
        const uint32_t pt = base + L::kOffP + slot * L::kQBytes, psf = base + L::kOffSFP + slot * 1024;
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) tc_cp_sf(sfv + 4 * ks, vsf + 512 * ks);
        ok = mbar_wait(bar(L::kPFull + slot), (li / kDepth) & 1, wc, kDPFull);
        if (!ok) break;
        tc_fence_after_sync();
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) tc_cp_sf(sfp + 4 * ks, psf + 512 * ks);
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
          mma_nvf4(tmem + TM::kO, make_desc_sw64(vt + 32 * ks), make_desc_sw64(pt + 32 * ks), idesc,
                   sfv + 4 * ks, sfp + 4 * ks, (li > 0 || ks > 0) ? 1u : 0u);
        }
        tc_commit(bar(L::kPvDone + slot));   // O stable; also: the P slot and the V stage are free
      }
      if (!ok) {
        const uint64_t t0 = globaltimer_ns();
        tc_commit(bar(L::kDrain + 1));
        while (!mbar_try_wait(bar(L::kDrain + 1), 0) && globaltimer_ns() - t0 < 50ull * 1000 * 1000) {}
      }
    }
  } else if (warp < 4 || warp >= 8) {
    // ============================================ softmax warpgroups, epilogue ==================
    // Warpgroup wg takes the blocks li = wg, wg + kWgs, ...; the first one also prepares the operands
    // and writes the result.  What a block hands to the next one is the reference maximum of its rows,
    // from warp wq of one warpgroup to warp wq of the other (every warp knows all rows); everything
    // else of a block -- about 1000 clocks of latencies -- then runs beside the neighbouring block's.
    const int wg = warp < 4 ? 0 : (warp >> 2) - 1, wq = warp & 3;
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>(wq * 32) << 16);
    s_red += wg * (2 * 4 * kMaxRows);
    uint32_t sync_phase = 0;
    // rendezvous of the 128 threads on an mbarrier (bounded, unlike bar.sync)
#define FA4_DEC_SYNC()                                                                          \
  mbar_arrive(bar(L::kSync + wg));                                                       \
  ok = __all_sync(0xffffffffu, mbar_wait(bar(L::kSync + wg), sync_phase & 1, wc, kDSync)); \
  sync_phase += 1;

    // ---- set-up: Q^T operand (rows x 64 bytes, rows past R zero), its scale chunks, zeroed
    //      P^T tiles and scale chunks (rows past R are never written again)
    ok = true;
    if (wg == 0) {
      for (uint32_t i = tid; i < (L::kOffRed - L::kOffQ) / 16; i += 128) {
        *reinterpret_cast<uint4*>(gbase + L::kOffQ + i * 16) = make_uint4(0u, 0u, 0u, 0u);  // Q, SFQ, P, SFP are contiguous
      }
      FA4_DEC_SYNC()
      if (ok) {
        const int r = tid >> 2, ch = tid & 3;
        if (r < R) *reinterpret_cast<uint4*>(gbase + L::kOffQ + sw64_offset(r, ch)) = q_pref;
      }
      if (ok && tid < 64) {
        // scale bytes of row r: two words (one per 64-element step) of the tiled layout
        const int r = tid >> 1, ks = tid & 1;
        if (r < R) *reinterpret_cast<uint32_t*>(gbase + L::kOffSFQ + 512 * ks + r * 16) = qsf_pref;
      }
      fence_proxy_async_smem();
      mbar_arrive(bar(L::kQReady));
    }

    // After the transpose below a thread owns ONE query row (row = lane % kR) with kR neighbouring
    // keys of its warp's 32 (group = lane / kR), so everything per row -- mask limit, reference
    // maximum, block exponent, running sum -- is scalar per thread and runs once per block, where a
    // thread that kept "its key, all rows" ran it kR times.
    const int my_row = lane & (kR - 1), grp = lane / kR;
    const int key_in_blk = wq * 32 + grp * kR;   // first of this thread's kR keys inside the block
    // Row sums: kStrands of them, that of block li in strand li % kStrands, each relative to the reference of its own
    // last block; so a row's sum is the same bits with two warpgroups and with four.  With two, a thread has two,
    // of which shared memory keeps the one that is not in use.
    float m_ref = kNegInf, l_sum = 0.f;
    float m_top = kNegInf;       // kBalanced: the highest reference so far (a warpgroup sees its own and those handed to it: all)
    static_assert(!kBal || kWgs <= 2, "every reference passes through every warpgroup");
    float2* strands = reinterpret_cast<float2*>(gbase + L::kOffSum) + wg * 128 + (tid & 127);    // [2][256]
    if (kOwn == 2) strands[0] = strands[256] = make_float2(0.f, kNegInf);
    // last visible key of the row (causal: bottom-right aligned on the entry's key count); rows
    // past R see nothing
    int lim = -1;
    if (my_row < R) {
      const int c = sk - p.Sq + fast_div(my_row, p.div_group);
      lim = (p.causal && c < sk - 1) ? c : sk - 1;
    }

    for (int li = wg; ok && li < n; li += kWgs) {
      const int nb = kBal && pre != 0 && li == 0 ? work.i0 - work.into : i0 + li;
      const uint32_t buf = li % kDepth, slot = li % kDepth;
      ok = __all_sync(0xffffffffu, mbar_wait(bar(L::kSFull + buf), (li / kDepth) & 1, wc, kDSFull));
      if (!ok) break;
      tc_fence_after_sync();
      float x[kR];
      tmem_ld_cols<kR>(lane_addr + TM::kS + kN * buf, reinterpret_cast<uint32_t*>(x));
      tc_wait_ld();
      tc_fence_before_sync();
      mbar_arrive(bar(L::kSFree + buf));

      // (key = lane, all rows) -> (row = lane % kR, kR keys): x[j] = score of key key_in_blk + j
      lane_group_transpose<kR>(x, lane);
      const int key0 = nb * kBlockN + key_in_blk;
      // kB 16-key blocks per thread: one (shared with neighbouring lanes) up to 16 rows, two of
      // its own in the 32-row form, where a thread owns all 32 keys of its warp
      constexpr int kB = kR <= 16 ? 1 : 2, kPer = kR / kB;
      float bm[kB];
#pragma unroll
      for (int q = 0; q < kB; ++q) {
        bm[q] = kNegInf;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
          x[q * kPer + j] = (key0 + q * kPer + j <= lim) ? x[q * kPer + j] : kNegInf;
          bm[q] = fmaxf(bm[q], x[q * kPer + j]);
        }
      }
      // maximum of the row's 16-key block (kept for the P scale), then of the warp's 32 keys
      float wm;
      if constexpr (kB == 1) {
#pragma unroll
        for (int o = kR; o < 16; o <<= 1) bm[0] = fmaxf(bm[0], __shfl_xor_sync(0xffffffffu, bm[0], o));
        wm = fmaxf(bm[0], __shfl_xor_sync(0xffffffffu, bm[0], 16));
      } else {
        wm = fmaxf(bm[0], bm[kB - 1]);
      }
      volatile float* red = s_red + ((li / kWgs) & 1) * (4 * kMaxRows);
      if (lane < kR) red[wq * kMaxRows + lane] = wm;
      FA4_DEC_SYNC()
      if (!ok) break;

      // reference maximum of the row (CTA-uniform per row: every warp computes the same value)
      const float m_loc = fmaxf(fmaxf(red[my_row], red[kMaxRows + my_row]),
                                fmaxf(red[2 * kMaxRows + my_row], red[3 * kMaxRows + my_row]));
      float m_prev = m_ref;
      if (kWgs > 1 && li > 0) {
        const int before = (wg + kWgs - 1) % kWgs;
        // the reference after block li - 1 (the unbroken chain also orders the reuse of the slots: block
        // li + 1 overwrites this one's source only after it has read what this block hands on)
        ok = __all_sync(0xffffffffu, mbar_wait(bar(L::kHand + 4 * before + wq), ((li - 1) / kWgs) & 1, wc, kDHand));
        if (!ok) break;
        m_prev = s_hand[(before * 4 + wq) * kMaxRows + my_row];
      }
      float m_new = next_reference(m_prev, m_loc, sc.sl2);
      if constexpr (kBal) {
        while (next_start < li) next_start += work.share;
        if (next_start == li) {
          // A split starts: its reference is the maximum of this block, up to kMaxFall below the highest one (further
          // down, or where the row sees no key, the one before stays).
          m_new = m_prev == kNegInf || (fmaxf(m_top, m_prev) - m_loc) * sc.sl2 <= kMaxFall ? m_loc : m_prev;
        }
        m_top = fmaxf(m_top, fmaxf(m_prev, m_new));
        if (pre != 0 && li == 0) {
#pragma unroll
          for (int j = 0; j < kR; ++j) x[j] = kNegInf;
        }
      }
      if (kWgs > 1) {
        if (lane < kR) s_hand[(wg * 4 + wq) * kMaxRows + my_row] = m_new;
        mbar_arrive(bar(L::kHand + 4 * wg + wq));
      }
      float fac = 1.f;
      bool moved_row = false;
      if (m_new != m_prev) {
        fac = reference_factor(m_prev, m_new, sc.sl2);
        moved_row = m_prev != kNegInf;
      }
      // the row sum of this block's strand follows the reference (kWgs = 1: by the same factor)
      if constexpr (kOwn == 2) {
        const float2 strand = strands[128 * (li & 2)];
        l_sum = strand.x;
        m_ref = strand.y;
      }
      if (m_new != m_ref) {
        l_sum *= kWgs == 1 ? fac : reference_factor(m_ref, m_new, sc.sl2);
        m_ref = m_new;
      }
      const bool moved = __any_sync(0xffffffffu, moved_row);   // every warp holds all rows

      // P slot free once P V of block li - kDepth has run
      if (li >= kDepth) {
        ok = __all_sync(0xffffffffu, mbar_wait(bar(L::kPvDone + slot), ((li - kDepth) / kDepth) & 1, wc,
                                               kDPvDone));
        if (!ok) break;
      }
      {
        float noff[kB];
        uint32_t ue[kB];
        float pv[kR];
#pragma unroll
        for (int q = 0; q < kB; ++q) {
          block_exponent1(bm[q], m_ref, sc.sl2, noff[q], ue[q]);
          float psum = 0.f;
#pragma unroll
          for (int j = 0; j < kPer; ++j) {
            pv[q * kPer + j] = ex2_approx(fmaf(x[q * kPer + j], sc.sl2, noff[q]));
            psum += pv[q * kPer + j];
          }
          l_sum = fmaf(psum, __uint_as_float(ue[q] << 23), l_sum);
        }
        if (kOwn == 2) strands[128 * (li & 2)] = make_float2(l_sum, m_ref);
        if (my_row < R) {   // rows past R stay zero (written once at set-up)
          // kR keys = kR / 2 bytes of the row's 64, inside one 16-byte chunk of the swizzled tile
          const uint32_t col = static_cast<uint32_t>(key_in_blk) >> 1;
          uint8_t* dst = gbase + L::kOffP + slot * L::kQBytes + sw64_offset(my_row, col >> 4) + (col & 15);
          // scale byte of 16-key block blk = key_in_blk / 16: chunk blk / 4, the row's word, byte blk % 4
          uint8_t* sf_dst = gbase + L::kOffSFP + slot * 1024 + 512 * (key_in_blk >> 6) + my_row * 16 +
                            ((key_in_blk >> 4) & 3);
          if constexpr (kR == 4) {
            *reinterpret_cast<uint16_t*>(dst) =
                static_cast<uint16_t>(pack2_e2m1(pv[0], pv[1]) | (pack2_e2m1(pv[2], pv[3]) << 8));
          } else if constexpr (kR == 8) {
            *reinterpret_cast<uint32_t*>(dst) = pack8_e2m1(pv[0], pv[1], pv[2], pv[3], pv[4], pv[5], pv[6], pv[7]);
          } else if constexpr (kR == 16) {
            *reinterpret_cast<uint2*>(dst) =
                make_uint2(pack8_e2m1(pv[0], pv[1], pv[2], pv[3], pv[4], pv[5], pv[6], pv[7]),
                           pack8_e2m1(pv[8 % kR], pv[9 % kR], pv[10 % kR], pv[11 % kR], pv[12 % kR], pv[13 % kR],
                                      pv[14 % kR], pv[15 % kR]));
          } else {
            uint32_t w[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              w[c] = pack8_e2m1(pv[(8 * c) % kR], pv[(8 * c + 1) % kR], pv[(8 * c + 2) % kR], pv[(8 * c + 3) % kR],
                                pv[(8 * c + 4) % kR], pv[(8 * c + 5) % kR], pv[(8 * c + 6) % kR], pv[(8 * c + 7) % kR]);
            }
            *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
          }
          if constexpr (kB == 2) {
            // the thread's two blocks are neighbours in the scale word of its row
            *reinterpret_cast<uint16_t*>(sf_dst) =
                static_cast<uint16_t>(((ue[0] - 0x78u) << 3) | (((ue[kB - 1] - 0x78u) << 3) << 8));
          } else if ((key_in_blk & 15) == 0) {
            *sf_dst = static_cast<uint8_t>((ue[0] - 0x78u) << 3);
          }
        }
      }

      // correction (rare): O^T holds the earlier blocks relative to the old references; here a
      // thread is a dv lane with all rows in its columns, the factor of row r sits in lane r
      if (li > 0 && moved) {
        ok = __all_sync(0xffffffffu, mbar_wait(bar(L::kPvDone + ((li - 1) % kDepth)),
                                               ((li - 1) / kDepth) & 1, wc, kDPvDone));
        if (!ok) break;
        tc_fence_after_sync();
        float o[kR];
        tmem_ld_cols<kR>(lane_addr + TM::kO, reinterpret_cast<uint32_t*>(o));
        tc_wait_ld();
#pragma unroll
        for (int r = 0; r < kR; ++r) o[r] *= __shfl_sync(0xffffffffu, fac, r);
        tmem_st_cols<kR>(lane_addr + TM::kO, reinterpret_cast<const uint32_t*>(o));
        tc_wait_st();
      }
      fence_proxy_async_smem();
      tc_fence_before_sync();
      mbar_arrive(bar(L::kPFull + slot));
    }

    // ---- epilogue: row sums over the 128 key lanes, then thread = dv lane of O^T --------------
    if (ok) {
      // this thread's share of its row; the lanes of one row are kR apart
      float v = l_sum;
#pragma unroll
      for (int o = kR; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if constexpr (kOwn == 2) {
        // the strand that is not the last block's (its index: that of the block before, two warpgroups ago)
        const int c = (n + kWgs - 1 - wg) / kWgs;
        const float2 other = strands[256 * (c & 1)];
        float v_old = other.x;
#pragma unroll
        for (int o = kR; o < 32; o <<= 1) v_old += __shfl_xor_sync(0xffffffffu, v_old, o);
        if (lane < kR) {
          s_old[(wg * 5 + wq) * kN + lane] = v_old;
          if (wq == 0) s_old[(wg * 5 + 4) * kN + lane] = other.y;
        }
      }
      // (the buffer of the exchange after the last one)
      volatile float* red = s_red + (((n + kWgs - 1 - wg) / kWgs) & 1) * (4 * kMaxRows);
      if (lane < kR) red[wq * kMaxRows + lane] = v;
      if (kWgs > 1 && wg > 0) {
        // the other warpgroups leave their sums and the references to the first and are done (the last reference in this
        // warp's own slot: what its last block handed on there, or -inf if it had none.  Another warp's slot
        // may not have been read yet: a warp of the next warpgroup can be a block behind this one)
        if (wq == 0 && lane < kR) s_hand[(wg * 4 + wq) * kMaxRows + lane] = m_ref;
        mbar_arrive(bar(L::kFin));
      } else {
        FA4_DEC_SYNC()
      }
    }
    if (ok && wg == 0) {
      if (kWgs > 1) ok = __all_sync(0xffffffffu, mbar_wait(bar(L::kFin), 0, wc, kDFin));
      // Per row, the lanes of a row alike: the sum over the warps in a fixed order (it does not depend on
      // timing), brought to the last reference of the row; the factor of the output; the LSE
      float scale = 0.f, lse = kNegInf;
      [[maybe_unused]] float back = 1.f;
      [[maybe_unused]] bool fell = false;
      if (ok) {
        float m_s[kStrands], l_s[kStrands], m_fin = kNegInf, l_tot = 0.f;
        [[maybe_unused]] float m_last = kNegInf;       // kBalanced: the last reference, that of O
#pragma unroll
        for (int i = 0; i < kStrands; ++i) {
          // strand i is one of warpgroup w, which did c blocks: that of its last block, with the sums in the buffer of
          // the exchange after the last one, or the other one
          const int w = i % kWgs, c = (n + kWgs - 1 - w) / kWgs;
          const bool last = kOwn == 1 || ((c + 1) & 1) == i / kWgs;
          volatile float* sum = (last ? s_red + (2 * w + (c & 1)) * (4 * kN) : s_old + w * (5 * kN)) + my_row;
          l_s[i] = ((sum[0] + sum[kN]) + sum[2 * kN]) + sum[3 * kN];
          const float handed = s_hand[w * 4 * kN + my_row];
          m_s[i] = !last ? s_old[(w * 5 + 4) * kN + my_row] : (w == 0 ? m_ref : handed);
          m_fin = fmaxf(m_fin, m_s[i]);
          if constexpr (kBal) m_last = i == (n - 1) % kStrands ? m_s[i] : m_last;
        }
        if constexpr (kBal) {
          // the sum goes to the highest reference, where it is of ordinary size; so does O, below
          m_fin = fmaxf(m_fin, m_top);
          back = reference_factor(m_last, m_fin, sc.sl2);
          fell = m_last != m_fin;
        }
#pragma unroll
        for (int i = 0; i < kStrands; ++i) l_tot = fmaf(l_s[i], reference_factor(m_s[i], m_fin, sc.sl2), l_tot);
        if (l_tot > 0.f && n > 0) scale = sc.out_scale / l_tot;
        lse = finish_lse(m_fin, l_tot, sc.sl2);
      }
      float o[kR];
#pragma unroll
      for (int r = 0; r < kR; ++r) o[r] = 0.f;
      if (ok && n > 0) {
        ok = __all_sync(0xffffffffu, mbar_wait(bar(L::kPvDone + ((n - 1) % kDepth)),
                                               ((n - 1) / kDepth) & 1, wc, kDPvDone));
        if (ok) {
          tc_fence_after_sync();
          tmem_ld_cols<kR>(lane_addr + TM::kO, reinterpret_cast<uint32_t*>(o));
          tc_wait_ld();
          if (kBal && __any_sync(0xffffffffu, fell)) {
#pragma unroll
            for (int r = 0; r < kR; ++r) o[r] *= __shfl_sync(0xffffffffu, back, r);
          }
        }
      }
      if (ok) {
        // (kMerge: the K and V rings are free, every product has completed)
        float* dst = reinterpret_cast<float*>(gbase + L::kOffK) + tid;
        constexpr int step = 128;
        if constexpr (kBal) {
          dst = d.o_partial + (int64_t)blockIdx.x * R * 128 + tid;
        } else if constexpr (!kMerge) {
          // row r = s * group + (head in the group): the rows of one token are neighbours
          dst = d.o_partial + ((((int64_t)split * p.B + b) * p.Sq) * p.Hq + hk * p.group) * 128 + tid;
        }
        int in_group = 0;
        if (kBal && work.pieces == 1) {
          // the result itself
          __nv_bfloat16* res = p.out + b * p.o_stride_b + (int64_t)hk * p.group * p.o_stride_h + tid;
#pragma unroll
          for (int r = 0; r < kR; ++r) {
            const float v = o[r] * __shfl_sync(0xffffffffu, scale, r);
            if (r < R) *res = __float2bfloat16_rn(v);
            res += p.o_stride_h;
            if (++in_group == p.group) {
              in_group = 0;
              res += p.o_stride_s - (int64_t)p.group * p.o_stride_h;
            }
          }
        } else
#pragma unroll
        for (int r = 0; r < kR; ++r) {
          if (r < R) *dst = o[r] * __shfl_sync(0xffffffffu, scale, r);   // lane r of every warp owns row r
          dst += step;
          if constexpr (!kMerge && !kBal) {
            if (++in_group == p.group) {
              in_group = 0;
              dst += (int64_t)(p.Hq - p.group) * 128;
            }
          }
        }
        if (tid < R) {
          if constexpr (kMerge) {
            reinterpret_cast<float*>(gbase + L::kOffV)[tid] = lse;
          } else {
            const int s = fast_div(tid, p.div_group), h = hk * p.group + tid - s * p.group;
            if (kBal && work.pieces > 1) d.lse_partial[(int64_t)blockIdx.x * R + tid] = lse;
            else if (!kBal) d.lse_partial[(((int64_t)split * p.B + b) * p.Hq + h) * p.Sq + s] = lse;
            else if (p.lse != nullptr) p.lse[((int64_t)b * p.Hq + h) * p.Sq + s] = lse;
          }
        }
      }
    }
#undef FA4_DEC_SYNC
  }

  if constexpr (kMerge) {
    // Merge (the arithmetic of combine_splits_kernel): row r by CTA r % splits, a warp a row, four dv a lane.  A launch of
    // its own for it costs 2-3 us behind a kernel of 6.  Every thread of every CTA comes here, also
    // after a wait that ran out (then nothing is written).
    cluster_sync();
    if (warp < 4) {
      const uint32_t ns = d.num_splits;
      const uint32_t gave_up = lane < ns ? ld_cluster_u32(base + L::kOffMisc + 4, lane) : 0u;
      const bool whole = !__any_sync(0xffffffffu, gave_up != 0u);
#pragma unroll 1
      for (int r = split + warp * ns; r < R && whole; r += 4 * ns) {
        float l[kMaxCluster], m = kNegInf;
        float4 v[kMaxCluster];
#pragma unroll
        for (uint32_t i = 0; i < kMaxCluster; ++i) {
          l[i] = kNegInf;
          v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (i < ns) {
            l[i] = __uint_as_float(ld_cluster_u32(base + L::kOffV + 4 * r, i));
            v[i] = ld_cluster_f4(base + L::kOffK + 16 * (r * 32 + lane), i);
          }
        }
#pragma unroll
        for (int i = 0; i < kMaxCluster; ++i) m = fmaxf(m, l[i]);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        float sum = 0.f;
        if (m != kNegInf) {
#pragma unroll
          for (int i = 0; i < kMaxCluster; ++i) {
            const float w = __expf(l[i] - m);
            sum += w;
            acc.x = fmaf(w, v[i].x, acc.x);
            acc.y = fmaf(w, v[i].y, acc.y);
            acc.z = fmaf(w, v[i].z, acc.z);
            acc.w = fmaf(w, v[i].w, acc.w);
          }
          const float inv = 1.f / sum;
          acc.x *= inv; acc.y *= inv; acc.z *= inv; acc.w *= inv;
        }
        const int s = fast_div(r, p.div_group), h = hk * p.group + r - s * p.group;
        *reinterpret_cast<uint2*>(p.out + b * p.o_stride_b + s * p.o_stride_s + h * p.o_stride_h + 4 * lane) =
            make_uint2(pack_bf16x2(acc.x, acc.y), pack_bf16x2(acc.z, acc.w));
        if (lane == 0 && p.lse != nullptr)
          p.lse[((int64_t)b * p.Hq + h) * p.Sq + s] = m == kNegInf ? kNegInf : m + __logf(sum);
      }
    }
    cluster_sync();      // no CTA leaves while another may read its shared memory
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 5) tmem_dealloc(tmem, TM::kCols);
}

}  // namespace fa4
