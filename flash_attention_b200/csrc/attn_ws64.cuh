// Warp-specialised kernel with 64-key sub-blocks and FOUR score buffers: every prefill call but split-KV,
// which stays with attn_ws.cuh.
//
// The kernel of attn_ws.cuh keeps two 128-column S buffers in tensor memory and lets two pairs of
// softmax warpgroups alternate over the 128-key blocks, a thread owning half a row.  The two
// warpgroups of a pair move in lockstep, so a scheduler sees only two independent softmax
// "strands", each with ~1000 clocks of exponentials and ~2000 clocks of latency-bound prologue /
// epilogue per block: the exponential unit idles ~40 % of the time, and every tile end drains
// the pipeline while the softmax warps read the accumulator out.
//
// Here a K/V block of 128 keys is processed as two sub-blocks of 64 keys, S has four buffers of 64
// columns (the same 256 tensor-memory columns), and each of the four softmax warpgroups owns one
// buffer: a thread holds the 64 scores of one WHOLE row of one sub-block -- the same register
// footprint -- so it takes the maxima itself (no statistics warpgroup), and the four warpgroups
// are independent strands at different phases.
//
//   warps 0-15  softmax: warpgroup w takes the sub-blocks with running index J % 4 == w; the
//               running reference maximum of a row is handed from the warpgroup of sub-block
//               J - 1 to that of J through shared memory
//   warp 16     TMA loads of Q (double buffered) and K (ring of 128-key tiles)
//   warp 17     Q K^T issuer: per K tile its scales to tensor memory and one N = 128 product into two neighbouring S
//               buffers
//   warp 18     P V issuer: per sub-block one K = 64 step into O, the scales of V and P before it
//   warp 19     TMA loads of V (its own ring)
//   warps 20-23 epilogue: combine the partial row sums, read O out, TMA store, LSE -- while the
//               softmax warpgroups already work on the next tile
//
// Sub-block j of a tile (visit order): keys 64 j .. 64 j + 63, ascending.  (The 128-key kernel
// visits the last visible block first; with 64-key steps that order makes the first references
// of a causal tile rest on one or two keys, and with the small lazy threshold that NVFP4 block
// scales allow nearly every tile then pays several accumulator corrections, each of which
// drains the P V pipeline.  Ascending, the first sub-block is fully visible.)
//
// Short tiles go through all of this code once per tile, 24 warps at their own places in it, and an SM's instruction
// cache holds about 32 KB: a 127-key window that visits two blocks a tile ran at 81 us with 49 KB of kernel and 400 k
// cache misses, and at 103 with work taken OUT by code that made it 1.4 M.  So what is rare is kept out of the loops
// (the soft cap has its own instantiations), and nothing is unrolled that runs once per tile.
// J = 2 * (blocks before this tile) + j selects buffers, P slots and barrier phases.  Operand
// formats, P quantisation, lazy reference and bounded waits are those of attn_ws.cuh.
#pragma once
#include "attn_ws.cuh"

namespace fa4 {
namespace ws64 {

constexpr int kStagesK = 4, kStagesV = 4;  // 128-key tiles
constexpr int kSBufs = 4;                  // S buffers of 64 columns
constexpr int kPSlots = 8;                 // P tiles of 64 keys (4 KB each)
constexpr int kThreads = 768;
constexpr int kLoadKWarp = 16, kIssuerWarp = 17, kPvIssuerWarp = 18, kLoadVWarp = 19, kEpilogueWarp0 = 20;
// Registers are a per-scheduler resource: 16384 per SM sub-partition, warp w living on sub-partition
// w % 4.  With 21-24 warps a sub-partition holds 6, so the launch gets 80 registers per thread and
// the CTA's pool per sub-partition is 6 x 32 x 80 = 15360.  setmaxnreg.inc draws from that pool
// (NOT from the whole register file) and blocks until it can be served: a budget above the pool
// never returns.  Per sub-partition: four softmax warps at 96, one service warp at 40 and one
// epilogue warp at 56 use exactly the pool.
constexpr int kRegsSoftmax = 96, kRegsOther = 40, kRegsEpilogue = 56, kRegsLaunch = 80;
// (Head dim 192, whose loader and Q K^T issuer hold three steps' worth of addresses: both at 48; B=8, S=2048,
// H=16 126.9 -> 123.8 us.  The other head dims lose 0.3 % that way.)
constexpr int kRegsEven = 48;
static_assert(2 * kRegsEven <= kRegsOther + kRegsEpilogue, "register pool of a sub-partition");
static_assert(kThreads == 768, "six warps per sub-partition");
static_assert(4 * kRegsSoftmax + kRegsOther + kRegsEpilogue <= 6 * kRegsLaunch,
              "register pool of a sub-partition");
static_assert((kThreads / 128) * 32 * kRegsLaunch <= 16384, "register file of a sub-partition");

// tensor memory: S[4] x 64 columns, O 128, scale factors
// (O at column 256 and Q scales at 384 as in the 128-key kernel); K and V scales have one slot of
// columns per shared-memory stage, written by the issuer in front of the first product that reads it (one
// thread, one pipe: no barrier).  us, copied by the loaders behind a barrier of their own -> by the issuers: 127-key
// window 81.5 -> 78.7, 24 packed sequences 174 -> 168.  In the plain form, both measured on the same day: 54 sequences
// of 300 45.5 -> 44.5 causal, 57.9 -> 55.6 not; 16 of 1024 62.3 -> 60.9; head dim 64, S = 16384 1277 -> 1270; but long tiles of
// head dim 128 lose 0.1-0.2 % (causal GQA 1310.5 -> 1312.2, S = 32768 10094 -> 10110), for which a second way of
// feeding the issuers is not kept.
// (sized for head dim 192: three 64-element steps, 12 scale columns per Q / K tile)
constexpr uint32_t kTmS64 = 0, kTmSFQ64 = 384 /* 12 */, kTmSFK64 = 396 /* 4 x 12 */, kTmSFV64 = 444 /* 4 x 8 */,
                   kTmSFP64 = 476 /* 4 x 4 */;
static_assert(kTmSFP64 + 16 <= 512, "tensor memory columns");
// shared-memory slots of a Q / K tile and of its scales, sized for head dim 192 (128 rows of 96
// bytes as three 32-byte-wide sub-tiles; three scale chunks)
constexpr uint32_t kQkSlot = 128 * 96, kQkSfSlot = 3 * 512;
constexpr uint64_t kDrainNs = 50ull * 1000 * 1000;   // limit of the waits for what is in flight when a CTA gives up
constexpr uint32_t kSlackNs = 500;         // suspend hint of the waits of roles with slack
constexpr uint32_t kPTileBytes = 128 * 32;  // 128 rows x 64 e2m1 keys
// P block scales of 64 keys that are all masked: 2^kEMin (powers of two: exponent e is byte (e + 7) << 3), or, in the
// form with a mantissa, the smallest scale it gives
constexpr uint32_t kMaskedScales = FA4_P_SCALE_E4M3 ? (uint32_t)(8 * kEMin + 56) * 0x01010101u : (uint32_t)((kEMin + 7) << 3) * 0x01010101u;

constexpr uint32_t kOffQ = 0;
constexpr uint32_t kOffK = kOffQ + 2 * kQkSlot;
constexpr uint32_t kOffV = kOffK + kStagesK * kQkSlot;
constexpr uint32_t kOffP = kOffV + kStagesV * kTileBytes;
constexpr uint32_t kOffSFQ = kOffP + kPSlots * kPTileBytes;
constexpr uint32_t kOffSFK = kOffSFQ + 2 * kQkSfSlot;
constexpr uint32_t kOffSFV = kOffSFK + kStagesK * kQkSfSlot;
constexpr uint32_t kOffSFP = kOffSFV + kStagesV * kSfBytes;      // kPSlots x 512
constexpr uint32_t kOffOut = kOffSFP + kPSlots * 512;            // 32 KB staging tile
constexpr uint32_t kOffHand = kOffOut + 32 * 1024;               // kSBufs x 128 reference maxima
constexpr uint32_t kOffFin = kOffHand + kSBufs * 128 * 4;        // 2 tiles x 4 WGs x 128 x (sum, ref)
constexpr uint32_t kOffTiles = kOffFin + 2 * 4 * 128 * 8;       // kMaxTiles records
constexpr uint32_t kOffBar = kOffTiles + kThreads * 32;

struct Bars {
  uint32_t base;
  static constexpr uint32_t kQFull = 0, kQEmpty = 2, kKFull = 4, kVFull = kKFull + kStagesK,
                            kKFree = kVFull + kStagesV, kVFree = kKFree + kStagesK,
                            kSFull = kVFree + kStagesV, kSFree = kSFull + kSBufs,
                            kHand = kSFree + kSBufs, kPFull = kHand + 4 * kSBufs, kPvDone = kPFull + kPSlots,
                            kFin = kPvDone + kPSlots, kFinFree = kFin + 2, kOFree = kFinFree + 2,
                            kDrain = kOFree + 1, kOFree2 = kDrain + 2, kOFull = kOFree2 + 1, kCount = kOFull + 2;
  __device__ explicit Bars(uint32_t b) : base(b) {}
  __device__ __forceinline__ uint32_t at(uint32_t idx) const { return base + 8u * idx; }
};
constexpr uint32_t kOffMisc = kOffBar + 8 * Bars::kCount;
constexpr uint32_t kSmemUsed = kOffMisc + 16 + sizeof(WaitCtx);
constexpr uint32_t kSmemRequest = kSmemUsed + 1024;
static_assert(kSmemRequest <= 227 * 1024, "shared memory");

enum Site64 {
  kS64QFull = 40, kS64QEmpty, kS64KFree, kS64VFree, kS64KFull, kS64VFull, kS64SFull, kS64SFree,
  kS64PFull, kS64PvDone, kS64Hand, kS64Fin, kS64FinFree, kS64FinalO, kS64OFree
};

// The tiles of this CTA, decoded once at kernel start -- one thread per tile -- into a table in shared
// memory that every role reads.  (Each of the seven roles used to decode every tile for itself: a few
// hundred instructions that ran in all 24 warps at every tile change and, being seven copies, pushed
// the rest of the kernel out of the instruction cache.)
struct alignas(16) TileRec {
  int m_blk, h, b;
  int n;          // K/V blocks this tile visits; 0: none is visible; -1: the tile has no rows at all (packed batch)
  int hk, sk;     // kv head; valid keys of the batch entry
  int off;        // row r of the tile sees keys up to off + r (plus the right window limit)
  int first;      // block the ascending visit starts at; negative: ~first, and the two blocks of the left edge last
};
static_assert(sizeof(TileRec) == 32, "two 16-byte loads");
constexpr int kMaxTiles = kThreads;   // per CTA and launch (the host launches longer lists in pieces)

// Visit order of a windowed tile: the i-th visited 128-key block.  Ascending from the first block
// the window reaches, EXCEPT that the two blocks at the window's left edge -- where the lower rows
// of the tile see a few keys or none, so that references taken there would be low -- are visited
// last: a tile starts at a block every row sees whole.  (The right edge, the diagonal, is last in
// ascending order anyway.)
__device__ __forceinline__ int window_visit_block(int i, const TileRec& t) {
  if (t.first >= 0) return t.first + i;
  const int lo = ~t.first;
  return i < t.n - 2 ? lo + 2 + i : lo + (i - (t.n - 2));
}
template <bool kGeneral>
__device__ __forceinline__ TileRec make_tile_rec(const KernelParams& p, int tile_idx) {
  const Tile t = decode_tile<kGeneral>(p, tile_idx);
  TileRec r;
  r.m_blk = t.m_blk;
  r.h = t.h;
  r.b = t.b;
  r.n = t.n_blocks;
  r.hk = t.hk;
  r.sk = key_len<kGeneral>(p, t);
  r.off = t.m_blk * kBlockM + r.sk - query_len<kGeneral>(p, t);
  r.first = t.nb_top - t.n_blocks + 1;
  if constexpr (kGeneral) {
    if (p.win_left >= 0 && r.n > 2 && r.off - p.win_left > 0) r.first = ~r.first;
    if (t.m_blk * kBlockM >= t.sq) r.n = -1;
  } else {
    r.first = 0;
  }
  return r;
}
// Packed batches: the list of the tiles that exist.  In a grid sized by the longest sequence most slots of
// a batch of unequal lengths are empty, and dealing slots to the CTAs leaves them with unequal work (24
// sequences of 32 to 2048 tokens: 23 % above the mean; dealt like this 1 %).  Sequences are ranked by their
// number of tiles; causal: last row blocks first, over the sequences that have them; otherwise the
// tiles of the longest sequence first.  All threads call it; `tile`: in: an index into this list; out: the
// index make_tile_rec takes for that tile (or -1).  Returns (end of the list, that index).  `mem`: 4
// kThreads words.  Out of line, so that the rest of the kernel's registers do not depend on it.
__device__ __noinline__ int2 live_tiles(const int32_t* cu_seqlens_q, int n, int num_m_blocks, int Hq, FastDiv div_hq,
                                        int causal, int tile, int tile_end, int* mem) {
  // tiles by sequence; then in ranked order: tiles, tiles of those ranked before, sequence
  int *count = mem, *sorted = mem + kThreads, *ahead = sorted + kThreads, *order = ahead + kThreads;
  const int tid = threadIdx.x, n4 = (n + 3) & ~3;
  int mine = 0;
  if (tid < n) {
    mine = (cu_seqlens_q[tid + 1] - cu_seqlens_q[tid] + kBlockM - 1) / kBlockM;
    mine = mine < 0 ? 0 : (mine < num_m_blocks ? mine : num_m_blocks);
  }
  if (tid < n4) count[tid] = mine;
  __syncthreads();
  int rank = 0, before = 0, total = 0;
#pragma unroll 2
  for (int j = 0; j < n4; j += 4) {
    const int4 c = *reinterpret_cast<const int4*>(count + j);
    const int v[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const bool first = v[k] > mine || (v[k] == mine && j + k < tid);
      rank += first ? 1 : 0;
      before += first ? v[k] : 0;
      total += v[k];
    }
  }
  if (tid < n) {
    sorted[rank] = mine;
    ahead[rank] = before;
    order[rank] = tid;
  }
  __syncthreads();
  if ((int64_t)total * Hq < tile_end) tile_end = total * Hq;
  if (tile >= tile_end) return make_int2(tile_end, -1);
  const int u = fast_div(tile, div_hq), h = tile - u * Hq;
  int m, r;
  if (causal) {
    // tiles in the row blocks above m: of the sequences with more than m + 1 tiles (the first c by rank),
    // all but m + 1 each
    auto above = [&](int m_blk) -> int {
      int c = 0, hi = n;
      while (c < hi) {
        const int mid = (c + hi) >> 1;
        if (sorted[mid] > m_blk + 1) c = mid + 1; else hi = mid;
      }
      return c == 0 ? 0 : ahead[c - 1] + sorted[c - 1] - c * (m_blk + 1);
    };
    int lo = 0, hi = num_m_blocks - 1;      // the smallest m with at most u tiles above it
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (above(mid) <= u) hi = mid; else lo = mid + 1;
    }
    m = lo;
    r = u - above(m);
  } else {
    int lo = 0, hi = n - 1;                   // the last rank that starts at or before u
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (ahead[mid] <= u) lo = mid; else hi = mid - 1;
    }
    r = lo;
    m = u - ahead[r];
  }
  return make_int2(tile_end, ((causal ? num_m_blocks - 1 - m : m) * n + order[r]) * Hq + h);
}
// Last visible key of row `row` inside block nb (>= 127: no mask), the first one, and whether any row of
// the tile needs a mask there (see causal_limit, lower_limit and block_needs_mask in attn_common.cuh).
template <bool kWindow>
__device__ __forceinline__ int upper_key(const KernelParams& p, const TileRec& t, int row, int nb) {
  const int len = t.sk - 1 - nb * kBlockN;
  if (!p.causal) return len;
  const int c = t.off + row + (kWindow ? p.win_right : 0) - nb * kBlockN;
  return c < len ? c : len;
}
__device__ __forceinline__ int lower_key(const KernelParams& p, const TileRec& t, int row, int nb) {
  return p.win_left < 0 ? -(1 << 30) : t.off + row - p.win_left - nb * kBlockN;
}
template <bool kWindow>
__device__ __forceinline__ bool needs_mask(const KernelParams& p, const TileRec& t, int nb) {
  const int k0 = nb * kBlockN;
  bool need = k0 + kBlockN > t.sk || (p.causal && k0 + kBlockN - 1 > t.off + (kWindow ? p.win_right : 0));
  if constexpr (kWindow) need = need || (p.win_left >= 0 && k0 < t.off + kBlockM - 1 - p.win_left);
  return need;
}

// byte offset of 16-byte chunk c (0, 1) of row r in a P tile (rows of 32 bytes, 32-byte swizzle)
__device__ __forceinline__ uint32_t sw32_offset(uint32_t row, uint32_t chunk) {
  return row * 32u + ((chunk ^ ((row >> 2) & 1u)) << 4);
}

}  // namespace ws64

// kD: head dimension of Q, K and V (128 or 64).  It sets the number of 64-element steps of Q K^T,
// the bytes of a Q / K tile (128 rows of kD / 2 bytes: 64-byte-swizzled rows for 128, 32-byte for
// 64) and of a V tile (kD rows of 128 keys), and the width of O.  Shared and tensor memory are
// laid out for 128 either way.
// kGeneral adds sliding windows (the block range starts at the first block the window reaches, both
// limits are masked), the learnable sink (one more term of the row sum, in the epilogue) and the
// soft cap (tanh on the raw scores); a compile-time switch so that the plain instantiation carries
// none of it.  The window instantiation also serves KV-cache views (per-entry key counts, page
// tables); split-KV stays with attn_ws.cuh.
// (kWindow separates the two halves of it: the window changes the tile geometry and the masks of
// the hot loop, sink and soft cap do not -- a call with only those keeps the plain geometry code,
// which measured 16 % faster than carrying the window arithmetic along.)
// kCache: per-entry key counts and page tables without the window arithmetic.
// kNarrow (windows of a few blocks): most visited blocks are masked and a tile is over after a handful of
// steps.  Masks go to the scores in registers instead of through tensor memory, which shortens the chain of a short
// tile and costs a long one, since the branch sits in the hot loop.  us, wide form -> this one: 127-key window, D = 64
// 83.6 -> 75.1; 1023 keys, D = 128 106.5 -> 108.5 (the line lies in api.cu).  Of the 75, by masks that pass over the
// 32-key halves a warp sees whole and a second accumulator, 69 are left.
template <int kD, bool kGeneral = false, bool kWindow = kGeneral, bool kCache = kWindow, bool kNarrow = false,
          bool kCap = false>
__global__ void __launch_bounds__(ws64::kThreads, 1)
attn_fwd_ws64_kernel(const __grid_constant__ CUtensorMap tm_q,
                     const __grid_constant__ CUtensorMap tm_k,
                     const __grid_constant__ CUtensorMap tm_v,
                     const __grid_constant__ CUtensorMap tm_o, const KernelParams p) {
  using namespace ws64;
  using ws::rescale_accumulator;
  using ws::mask_scores_in_tmem;
  using ws::stage_accumulator_chunk;
  using ws::tile_of_round;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gbase = smem_raw + (base - smem_u32(smem_raw));
  const Bars bars(base + kOffBar);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gbase + kOffMisc);
  volatile uint32_t* s_abort = reinterpret_cast<volatile uint32_t*>(gbase + kOffMisc + 4);
  volatile float* s_hand = reinterpret_cast<volatile float*>(gbase + kOffHand);  // [4][128]
  volatile float* s_fin = reinterpret_cast<volatile float*>(gbase + kOffFin);    // [2][4][128][2]

  const int tid = threadIdx.x;
  const int warp = warp_index();
  const int lane = tid & 31;
  WaitCtx& wc = *reinterpret_cast<WaitCtx*>(gbase + kOffMisc + 16);
  const int ncta = gridDim.x, cta = blockIdx.x;
  TileRec* s_tiles = reinterpret_cast<TileRec*>(gbase + kOffTiles);

  if (tid == 0) {
    *s_abort = 0u;
    wc = WaitCtx{s_abort, p.status, p.budget_ns, p.epoch};
    for (int b = 0; b < 2; ++b) {
      mbar_init(bars.at(Bars::kQFull + b), 1);
      mbar_init(bars.at(Bars::kQEmpty + b), 1);
    }
    for (int b = 0; b < 2; ++b) mbar_init(bars.at(Bars::kDrain + b), 1);
    for (int s = 0; s < kStagesK; ++s) {
      mbar_init(bars.at(Bars::kKFull + s), 1);
      mbar_init(bars.at(Bars::kKFree + s), 1);
    }
    for (int s = 0; s < kStagesV; ++s) {
      mbar_init(bars.at(Bars::kVFull + s), 1);
      mbar_init(bars.at(Bars::kVFree + s), 1);
    }
    for (int s = 0; s < kSBufs; ++s) {
      mbar_init(bars.at(Bars::kSFull + s), 1);
      mbar_init(bars.at(Bars::kSFree + s), 128);    // the softmax warpgroup that owns the buffer
      for (int q = 0; q < 4; ++q) mbar_init(bars.at(Bars::kHand + 4 * s + q), 32);  // per warp quarter
    }
    for (int s = 0; s < kPSlots; ++s) {
      mbar_init(bars.at(Bars::kPFull + s), 128);
      mbar_init(bars.at(Bars::kPvDone + s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bars.at(Bars::kFin + b), 512);      // the four softmax warpgroups
      mbar_init(bars.at(Bars::kFinFree + b), 128);  // the epilogue warpgroup
    }
    mbar_init(bars.at(Bars::kOFree), 128);
    if constexpr (kD == 64 && kNarrow) {            // two accumulators
      mbar_init(bars.at(Bars::kOFree2), 128);
      for (int b = 0; b < 2; ++b) mbar_init(bars.at(Bars::kOFull + b), 1);
    }
    fence_barrier_init();
  }
  if (warp == kLoadKWarp && lane == 0) {
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
  }
  if (warp == kLoadVWarp && lane == 0) tma_prefetch_desc(&tm_v);
  if (warp == kIssuerWarp) {
    tmem_alloc(base + kOffMisc, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  if constexpr (kWindow || kCache) pdl_wait();     // (their tiles depend on lengths in memory)
  // this CTA's tiles: p.tile_begin + tile_of_round(0), (1), ... below tile_end
  int tile_end = p.tile_end;
  {
    int tile = p.tile_begin + tile_of_round(tid, cta, ncta), list_end = tile_end;
    if constexpr (kWindow || kCache) {
      // (the P tiles' memory is free until the first scores)
      if (p.compact_tiles) {
        const int2 live = live_tiles(p.cu_seqlens_q, p.B, p.num_m_blocks, p.Hq, p.div_hq, p.causal, tile, tile_end,
                                     reinterpret_cast<int*>(gbase + kOffP));
        tile_end = live.x;
        tile = live.y >= 0 ? live.y : 0x7fffffff;
        list_end = 0x7fffffff;
      }
    }
    if (tile < list_end) s_tiles[tid] = make_tile_rec<kWindow || kCache>(p, tile);
  }
  if constexpr (!(kWindow || kCache)) pdl_wait();
  __syncthreads();
  tc_fence_after_sync();
  pdl_trigger();
  const uint32_t tmem = *tmem_slot;
  const ScoreScales sc = score_scales(p);
  static_assert(kD == 128 || kD == 64 || kD == 192, "head dimensions built: 128, 64 and (192, 128)");
  constexpr int kDv = kD == 192 ? 128 : kD;            // head dim of V and O
  constexpr uint32_t idesc_qk = make_idesc_nvf4(128, 128);
  constexpr uint32_t idesc_pv = make_idesc_nvf4(128, kDv);
  // Narrow windows at head dim 64 have tensor memory for two accumulators: P V of a tile, a handful of steps, does not
  // wait for the one before to be read out.  us, one -> two: 127-key window 72.1 -> 69.6.
  constexpr uint32_t kOBufs = kD == 64 && kNarrow ? 2 : 1;
  auto o_column = [&](uint32_t tile) -> uint32_t { return kTmO + 64 * (tile % kOBufs); };
  auto o_free = [&](uint32_t tile) -> uint32_t { return bars.at(tile % kOBufs ? Bars::kOFree2 : Bars::kOFree); };
  // Where the softmax step is cut for the compiler's scheduler.  Left as one piece, exponentials of a step can move up
  // among its maxima and hand-over, which the next warpgroup waits for; what kept them apart was a wait for
  // the P slot between the two, which now is the Q K^T issuer's.  Which cut pays differs by form.  us, wait / no cut /
  // in front of the exponentials / of the maxima / both:
  //   plain: causal GQA, B=2, S=8192 660 / 699 / 646 / 728 / 640, at D = 64 656 / 689 / 638 / 727 / 633
  //   D = 128: 24 packed sequences 166.6 / 163.9 / 166.1 / 215.5 / 167.6; 512 tokens against 32768 keys of a cache 199.5 / 196.0 /
  //     199.6 / 296 / 199.5; windows of 1023, 4096 keys 219.4 / 217.7 / 219.2 / 295 / 231.5, 565.9 / 564.8 / 567.7 / 844 / 578
  //   D = 64: 100 packed sequences 154.2 / 158.3 / 153.2 / 158.1 / 155.0, 8 long ones 168.2 / 182.5 / 165.6 / 177.0 / 166.6; windows
  //     of 1023, 16383 keys 212.0 / 208.8 / 207.5 / 220.8 / 212.7, 1388 / 1376 / 1352 / 1544 / 1387
  //   D = 192: 20 packed sequences 126.3 / 134.4 / 124.9 / 129.9 / 124.1, 60 short ones 72.5 / 74.4 / 72.0 / 73.9 / 72.8
  // Further cuts in the plain form: in front of the reference 643, between the maxima 643, in front of the last
  // stores 645, between the 16-key blocks 656 and 680.  (nvcc 12.9.86: what the scheduler does with a cut is the compiler's, so another one
  // wants these measured anew.  With the cuts the plain forms spill 12 bytes, at D = 64 20, without 0 and 12.)
  constexpr bool kPlain = !(kWindow || kCache);
  // The soft cap's forms (its 64 tanh stand in front of the maxima) take the first cut alone: plain, wait / first cut / both
  // 358 / 352 / 362, at D = 64 355 / 348 / 356, window of 1023 keys, wait / none / first 182 / 196 / 181.
  // The branch by which a row sum follows the reference, in front of the block exponents instead of behind them: 641 -> 637.8,
  // 633.6 -> 630.2 (D = 64), narrow windows 86.5 -> 84.7, 68.9 -> 68.4; the cache forms lose (packed 163.5 -> 164.9).
  constexpr bool kSumFirst = kPlain || kNarrow;
  constexpr bool kCutExp = !kNarrow && (kPlain || kD != 128 || kCap), kCutMax = kPlain && !kCap;
  constexpr int kSteps = kD / 64;                      // 64-element steps of Q K^T
  constexpr uint32_t kQkBytes = 128u * kD / 2;         // bytes of a Q or K tile
  constexpr uint32_t kQkSfBytes = kSteps * 512u;       // its scale chunks (128 rows x kD / 16)
  constexpr uint32_t kVBytes = kDv * 64u;              // V tile: kDv rows of 128 keys
  // A Q / K tile in shared memory: one 64-byte-swizzled box for head dim 128; for 64 and 192 one or
  // three 32-byte-wide boxes (32-byte swizzle, 4 KB each), one per 64-element step.
  auto load_qk_tile = [&](uint32_t dst, const CUtensorMap* tm, uint32_t bar, int h, int row, int b) {
    if constexpr (kD == 128) {
      tma_load_4d(dst, tm, bar, 0, h, row, b);
    } else {
#pragma unroll
      for (int j = 0; j < kSteps; ++j) tma_load_4d(dst + 4096 * j, tm, bar, 32 * j, h, row, b);
    }
  };
  auto desc_qk = [&](uint32_t tile, int j) -> uint64_t {
    if constexpr (kD == 128) return make_desc_sw64(tile + 32 * j);
    return make_desc_sw32(tile + 4096 * j);
  };

  // whole rounds, and the last partial one if it reaches this CTA
  const int num_rounds = (tile_end - p.tile_begin) / ncta +
                         (p.tile_begin + tile_of_round((tile_end - p.tile_begin) / ncta, cta, ncta) < tile_end ? 1 : 0);
#define FA4_FOR_EACH_TILE                                                                        \
  uint32_t gb = 0, ti = 0;                                                                       \
  bool ok = true;                                                                                \
  for (int it = 0; ok && it < num_rounds; ++it)

  if (warp >= kEpilogueWarp0) {
    // =========================================== epilogue warpgroup =============================
    // Thread = row.  Per tile: combine the four partial row sums, wait for the last P V, move O
    // from tensor memory to the staging tile (bf16, normalised), send it with TMA, write the LSE.
    // The softmax warpgroups meanwhile work on the next tile; only the P V issuer waits for the
    // accumulator to be read out.  Every warp stages and sends its own 32 rows: no rendezvous of the
    // four.
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kD == 192 ? kRegsEven : kRegsEpilogue));
    const int row = tid & 127;
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    if (warp == kEpilogueWarp0 && lane == 0) tma_prefetch_desc(&tm_o);
    FA4_FOR_EACH_TILE {
      const TileRec t = s_tiles[it];
      const int n = t.n;
      const int q_idx = t.m_blk * kBlockM + row;
      if constexpr (kWindow || kCache) {
        // a tile past the end of a short sequence of a packed batch has no rows at all
        if (n < 0) continue;
      }
      // the staging rows are free once the previous store has read them
      if (lane == 0) bulk_wait_group_read0();
      __syncwarp();
      float scale = 0.f, m_fin = kNegInf, l_tot = 0.f;
      if (n > 0) {
        const uint32_t fb = ti & 1;
        ok = __all_sync(0xffffffffu, mbar_wait_flag(bars.at(Bars::kFin + fb), (ti >> 1) & 1, s_abort));
        if (!ok) break;
        volatile float* fin_slot = s_fin + fb * (4 * 128 * 2);
        float lw[4], mw[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          lw[w] = fin_slot[(w * 128 + row) * 2];
          mw[w] = fin_slot[(w * 128 + row) * 2 + 1];
          m_fin = fmaxf(m_fin, mw[w]);
        }
        mbar_arrive(bars.at(Bars::kFinFree + fb));
#pragma unroll
        for (int w = 0; w < 4; ++w) l_tot += lw[w] * reference_factor(mw[w], m_fin, sc.sl2);
        if (m_fin == kNegInf) l_tot = 0.f;
        if constexpr (kGeneral) {
          // the sink joins the row sum, relative to the row's reference maximum
          if (p.sink != nullptr && m_fin != kNegInf) {
            l_tot += ex2_approx(static_cast<float>(kShift) + p.sink[t.h] * 1.4426950408889634f - m_fin * sc.sl2);
          }
        }
        const uint32_t Jl = 2 * gb + 2 * n - 1;
        // (with two accumulators the product that comes next to this P slot may be done before this wait begins, and
        // its barrier a phase further: the accumulator has one of its own)
        const uint32_t bar_o = kOBufs > 1 ? Bars::kOFull + ti % kOBufs : Bars::kPvDone + (Jl % kPSlots);
        ok = __all_sync(0xffffffffu, mbar_wait_flag(bars.at(bar_o), (kOBufs > 1 ? ti / kOBufs : Jl / kPSlots) & 1, s_abort));
        if (!ok) break;
        tc_fence_after_sync();
        scale = (l_tot > 0.f) ? sc.out_scale / l_tot : 0.f;
      }
      uint8_t* const out_row = gbase + kOffOut + row * 128;
      if (n == 0) {
#pragma unroll 1
        for (int v = 0; v < kDv / 8; ++v)
          *reinterpret_cast<uint4*>(out_row + (v >> 3) * (16 * 1024) + (v & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll 1
      for (int c = 0; c < (n > 0 ? kDv / 32 : 0); ++c) {
        uint8_t* box_row = out_row + (c >> 1) * (16 * 1024);
        uint32_t o[32];
        tmem_ld32(lane_addr + o_column(ti) + 32 * c, o);
        tc_wait_ld();
        if (c == kDv / 32 - 1) {
          tc_fence_before_sync();
          mbar_arrive(o_free(ti));  // the P V issuer may start the next tile
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          uint4 w;
          w.x = pack_bf16x2(__uint_as_float(o[8 * v + 0]) * scale, __uint_as_float(o[8 * v + 1]) * scale);
          w.y = pack_bf16x2(__uint_as_float(o[8 * v + 2]) * scale, __uint_as_float(o[8 * v + 3]) * scale);
          w.z = pack_bf16x2(__uint_as_float(o[8 * v + 4]) * scale, __uint_as_float(o[8 * v + 5]) * scale);
          w.w = pack_bf16x2(__uint_as_float(o[8 * v + 6]) * scale, __uint_as_float(o[8 * v + 7]) * scale);
          const int chunk = ((c & 1) * 4 + v) ^ (row & 7);
          *reinterpret_cast<uint4*>(box_row + chunk * 16) = w;
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      const bool packed = (kWindow || kCache) && p.cu_seqlens_q != nullptr;
      const int q0 = packed ? p.cu_seqlens_q[t.b] : 0;
      const int sq = packed ? p.cu_seqlens_q[t.b + 1] - q0 : p.Sq;
      const int row0 = t.m_blk * kBlockM + (warp & 3) * 32;     // first row of this warp
      if (packed && row0 + 32 > sq) {
        // last, partial rows of a packed sequence: a tiled store would run into the rows of the
        // next sequence (the tensor map only clips at the end of the whole batch), so every
        // thread copies its own row from the staging tile, if it has one
        if (q_idx < sq) {
          __nv_bfloat16* orow = p.out + (int64_t)(q0 + q_idx) * p.o_stride_s + (int64_t)t.h * p.o_stride_h;
#pragma unroll 1
          for (int c16 = 0; c16 < kDv / 8; ++c16) {
            const uint8_t* src = gbase + kOffOut + (c16 >> 3) * (16 * 1024) + row * 128 + (((c16 & 7) ^ (row & 7)) << 4);
            reinterpret_cast<uint4*>(orow)[c16] = *reinterpret_cast<const uint4*>(src);
          }
        }
      } else if (lane == 0 && row0 < sq) {
#pragma unroll
        for (int bx = 0; bx < kDv / 64; ++bx) {
          tma_store_4d(&tm_o, base + kOffOut + bx * 16 * 1024 + (warp & 3) * 4096, 64 * bx, t.h, q0 + row0,
                       packed ? 0 : t.b);
        }
        bulk_commit_group();
      }
      if (q_idx < sq && p.lse != nullptr) {
        float lse_v = finish_lse(m_fin, l_tot, sc.sl2);
        if constexpr (kGeneral) {
          // a row without visible keys still has its sink: LSE = sink, output zero
          if (p.sink != nullptr && m_fin == kNegInf) lse_v = p.sink[t.h];
        }
        if (packed) {
          p.lse[(int64_t)t.h * p.total_q + q0 + q_idx] = lse_v;   // (Hq, total_q)
        } else {
          p.lse[((int64_t)t.b * p.Hq + t.h) * p.Sq + q_idx] = lse_v;
        }
      }
      gb += n;
      ti += (n > 0) ? 1u : 0u;
    }
    if (lane == 0) bulk_wait_group0();
  } else if (warp >= kLoadKWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kD == 192 ? kRegsEven : kRegsOther));
    if ((warp == kLoadKWarp || warp == kLoadVWarp) && elect_one()) {
      // ========================================= TMA loaders ====================================
      // One warp streams Q and K, the other V, each as far ahead as its own ring allows: what Q K^T of
      // the next tile needs never queues behind a V stage that P V has yet to free.
      const bool is_k = warp == kLoadKWarp;
      const uint32_t full0 = is_k ? Bars::kKFull : Bars::kVFull, free0 = is_k ? Bars::kKFree : Bars::kVFree;
      uint32_t issued = 0, issued_q = 0;
      FA4_FOR_EACH_TILE {
        const TileRec t = s_tiles[it];
        const int n = t.n;
        if (n <= 0) continue;
        // a packed batch has no batch dimension: the sequence's first row is added to the row
        // coordinate instead (the scale tiles stay per sequence)
        const bool packed = (kWindow || kCache) && p.cu_seqlens_q != nullptr;
        int k0 = 0;      // first key of the sequence inside the packed tensor
        if (packed) k0 = !is_k && p.cu_seqlens_v != nullptr ? p.cu_seqlens_v[t.b] : p.cu_seqlens_k[t.b];
        if (is_k) {
          if (it > 0 && status_poisoned(p.status, p.epoch)) {
            // another CTA of this launch failed: stop this one quickly.  Only this role polls the
            // status word (a global load at every tile start but the first, whose loads it would hold up by its
            // latency); the others see the abort flag in their next wait, when the tiles stop coming
            *s_abort = 1u;
            break;
          }
          const uint32_t qb = ti & 1;
          if (ti >= 2) {
            ok = mbar_wait_relaxed<kSlackNs>(bars.at(Bars::kQEmpty + qb), ((ti - 2) >> 1) & 1, wc, kS64QEmpty);
            if (!ok) break;
          }
          mbar_arrive_expect_tx(bars.at(Bars::kQFull + qb), kQkBytes + kQkSfBytes);
          load_qk_tile(base + kOffQ + qb * kQkSlot, &tm_q, bars.at(Bars::kQFull + qb), t.h,
                       (packed ? p.cu_seqlens_q[t.b] : 0) + t.m_blk * kBlockM, packed ? 0 : t.b);
          bulk_load(base + kOffSFQ + qb * kQkSfSlot,
                    p.q_sf + t.b * p.qsf_stride_b + t.h * p.qsf_stride_h + (int64_t)t.m_blk * kQkSfBytes,
                    kQkSfBytes, bars.at(Bars::kQFull + qb));
          issued_q = ti + 1;
        }
        for (int i = 0; i < n; ++i) {
          const uint32_t G = gb + i, st = G % kStagesK;
          const int nb = kWindow ? window_visit_block(i, t) : i;  // ascending
          if (G >= kStagesK) {
            ok = mbar_wait_relaxed<kSlackNs>(bars.at(free0 + st), ((G - kStagesK) / kStagesK) & 1, wc,
                                             is_k ? kS64KFree : kS64VFree);
            if (!ok) break;
          }
          const uint32_t full = bars.at(full0 + st);
          mbar_arrive_expect_tx(full, is_k ? kQkBytes + kQkSfBytes : kVBytes + kSfBytes);
          // where logical K/V block nb of this batch entry lives: the entry itself, or (KV-cache views) a
          // page of the pool and the block in it
          int kb = t.b, nbl = nb;
          if constexpr (kWindow || kCache) {
            if (p.page_table != nullptr) {
              const int pg = fast_div(nb, p.div_page);
              kb = p.page_table[(int64_t)t.b * p.pages_per_seq + pg];
              nbl = nb - pg * (p.page_size / kBlockN);
            }
          }
          if (is_k) {
            load_qk_tile(base + kOffK + st * kQkSlot, &tm_k, full, t.hk, k0 + nbl * kBlockN, packed ? 0 : kb);
            bulk_load(base + kOffSFK + st * kQkSfSlot,
                      p.k_sf + kb * p.ksf_stride_b + t.hk * p.ksf_stride_h + (int64_t)nbl * kQkSfBytes, kQkSfBytes, full);
          } else {
            tma_load_4d(base + kOffV + st * kTileBytes, &tm_v, full, (k0 + nbl * kBlockN) / 2, 0, t.hk, packed ? 0 : kb);
            bulk_load(base + kOffSFV + st * kSfBytes,
                      p.v_sf + kb * p.vsf_stride_b + t.hk * p.vsf_stride_h + (int64_t)nbl * kSfBytes, kSfBytes, full);
          }
          issued = G + 1;
        }
        if (!ok) break;
        gb += n;
        ti += 1;
      }
      if (!is_k && ok && gb > 0) {
        // The epilogue's wait for a tile's last product has no clock (mbar_wait_flag).  Behind every other tile the
        // P V issuer waits for O; behind the last one this loader stays until the product has run.  (The same
        // wait in the P V issuer moved the compiler's code of the softmax loop: causal GQA 1428 -> 1436 us,
        // non-causal 711 -> 717, a 127-key window 92.4 -> 94.2; here 1431, 712, 92.1.)
        const uint32_t Jl = 2 * gb - 1;
        ok = mbar_wait_relaxed<kSlackNs>(bars.at(Bars::kPvDone + (Jl % kPSlots)), (Jl / kPSlots) & 1, wc, kS64FinalO);
      }
      if (!ok) {
        // bounded drain: let the copies already issued land before the CTA's memory is released
        const uint64_t t0 = globaltimer_ns();
        const uint64_t lim = kDrainNs;
        for (uint32_t i = issued > kStagesK ? issued - kStagesK : 0; i < issued; ++i) {
          while (!mbar_try_wait(bars.at(full0 + (i % kStagesK)), (i / kStagesK) & 1) && globaltimer_ns() - t0 < lim) {}
        }
        for (uint32_t i = issued_q > 2 ? issued_q - 2 : 0; i < issued_q; ++i) {
          while (!mbar_try_wait(bars.at(Bars::kQFull + (i & 1)), (i >> 1) & 1) && globaltimer_ns() - t0 < lim) {}
        }
      }
    } else if (warp == kIssuerWarp && elect_one()) {
      // ========================================= QK^T issuer ====================================
      FA4_FOR_EACH_TILE {
        const TileRec t = s_tiles[it];
        const int n = t.n;
        if (n <= 0) continue;
        const uint32_t qb = ti & 1;
        ok = mbar_wait(bars.at(Bars::kQFull + qb), (ti >> 1) & 1, wc, kS64QFull);
        if (!ok) break;
        tc_fence_after_sync();
        uint64_t dq[kSteps];
#pragma unroll
        for (int ks = 0; ks < kSteps; ++ks) {
          tc_cp_sf(tmem + kTmSFQ64 + 4 * ks, base + kOffSFQ + qb * kQkSfSlot + 512 * ks);
          dq[ks] = desc_qk(base + kOffQ + qb * kQkSlot, ks);
        }
        for (int i = 0; ok && i < n; ++i) {
          const uint32_t G = gb + i, st = G % kStagesK;
          ok = mbar_wait(bars.at(Bars::kKFull + st), (G / kStagesK) & 1, wc, kS64KFull);
          if (!ok) break;
          tc_fence_after_sync();
          const uint32_t sfk = tmem + kTmSFK64 + 12 * st;
          const uint32_t kt = base + kOffK + st * kQkSlot;
          // one product of N = 128 fills the two neighbouring S buffers of sub-blocks 2G and 2G + 1
          // (keys 0-63 and 64-127 of the tile): half the tcgen05 instructions of two N = 64
          // products, and the in-order issue slots of this thread are scarce
          const uint32_t J0 = 2 * G, b0 = J0 % kSBufs;  // 0 or 2
          // P of step J0 + 1 goes where P of step J0 + 1 - kPSlots is (and the softmax warps have no wait of their own for it)
          if (J0 >= kPSlots) {
            ok = mbar_wait(bars.at(Bars::kPvDone + ((J0 + 1) % kPSlots)), ((J0 + 1 - kPSlots) / kPSlots) & 1, wc, kS64PvDone);
            if (!ok) break;
          }
          if (J0 >= kSBufs) {
            ok = mbar_wait(bars.at(Bars::kSFree + b0), ((J0 - kSBufs) / kSBufs) & 1, wc, kS64SFree) &&
                 mbar_wait(bars.at(Bars::kSFree + b0 + 1), ((J0 - kSBufs) / kSBufs) & 1, wc, kS64SFree);
            if (!ok) break;
            tc_fence_after_sync();
          }
#pragma unroll
          for (int ks = 0; ks < kSteps; ++ks) tc_cp_sf(sfk + 4 * ks, base + kOffSFK + st * kQkSfSlot + 512 * ks);
#pragma unroll
          for (int ks = 0; ks < kSteps; ++ks) {
            mma_nvf4(tmem + kTmS64 + 64 * b0, dq[ks], desc_qk(kt, ks), idesc_qk,
                     tmem + kTmSFQ64 + 4 * ks, sfk + 4 * ks, ks > 0 ? 1u : 0u);
          }
          tc_commit(bars.at(Bars::kSFull + b0));  // both softmax warpgroups of the pair wait on it
          tc_commit(bars.at(Bars::kKFree + st));  // the K stage is free once both products have run
        }
        if (!ok) break;
        tc_commit(bars.at(Bars::kQEmpty + qb));
        gb += n;
        ti += 1;
      }
      if (!ok) {
        const uint64_t t0 = globaltimer_ns();
        tc_commit(bars.at(Bars::kDrain));
        while (!mbar_try_wait(bars.at(Bars::kDrain), 0) && globaltimer_ns() - t0 < kDrainNs) {}
      }
    } else if (warp == kPvIssuerWarp && elect_one()) {
      // ========================================= P V issuer =====================================
      FA4_FOR_EACH_TILE {
        const TileRec t = s_tiles[it];
        const int n = t.n;
        if (n <= 0) continue;
        for (int i = 0; ok && i < n; ++i) {
          const uint32_t G = gb + i, st = G % kStagesV;
          ok = mbar_wait(bars.at(Bars::kVFull + st), (G / kStagesV) & 1, wc, kS64VFull);
          if (!ok) break;
          tc_fence_after_sync();
          tc_cp_sf(tmem + kTmSFV64 + 8 * st, base + kOffSFV + st * kSfBytes);
          tc_cp_sf(tmem + kTmSFV64 + 8 * st + 4, base + kOffSFV + st * kSfBytes + 512);
          const uint32_t vt = base + kOffV + st * kTileBytes;
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            const uint32_t J = 2 * G + s, slot = J % kPSlots, tb = J % kSBufs;
            const uint32_t h64 = s;
            ok = mbar_wait(bars.at(Bars::kPFull + slot), (J / kPSlots) & 1, wc, kS64PFull);
            if (!ok) break;
            if (i == 0 && s == 0 && ti >= kOBufs) {
              // O of the tile before (the one before that) must have been copied out of tensor memory
              ok = mbar_wait(o_free(ti), ((ti - kOBufs) / kOBufs) & 1, wc, kS64OFree);
              if (!ok) break;
            }
            tc_fence_after_sync();
            const uint32_t sfp = tmem + kTmSFP64 + 4 * tb, sfv = tmem + kTmSFV64 + 8 * st + 4 * h64;
            tc_cp_sf(sfp, base + kOffSFP + slot * 512);
            mma_nvf4(tmem + o_column(ti), make_desc_sw32(base + kOffP + slot * kPTileBytes),
                     make_desc_sw64(vt + 32 * h64), idesc_pv, sfp, sfv, (i > 0 || s > 0) ? 1u : 0u);
            tc_commit(bars.at(Bars::kPvDone + slot));
          }
          if (!ok) break;
          tc_commit(bars.at(Bars::kVFree + st));
        }
        if (!ok) break;
        if (kOBufs > 1) tc_commit(bars.at(Bars::kOFull + ti % kOBufs));
        gb += n;
        ti += 1;
      }
      if (!ok) {
        const uint64_t t0 = globaltimer_ns();
        tc_commit(bars.at(Bars::kDrain + 1));
        while (!mbar_try_wait(bars.at(Bars::kDrain + 1), 0) && globaltimer_ns() - t0 < kDrainNs) {}
      }
    }
  } else {
    // =========================================== softmax warpgroups =============================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsSoftmax));
    const int wg = warp >> 2;                 // 0..3: owns S buffer wg, i.e. the sub-blocks J % 4 == wg
    const int row = (warp & 3) * 32 + lane;   // tile row == tensor-memory lane
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const uint32_t s_addr = lane_addr + kTmS64 + 64 * wg;

    // The running reference, handed from the warpgroup of sub-block J - 1 to that of J through shared memory (one
    // float per row).  Every sub-block but the CTA's very first waits for its predecessor's hand-over,
    // also the first one of a tile (which ignores the value): the unbroken chain is what orders
    // the reuse of a slot -- the value of sub-block J is overwritten by J + 4, which follows
    // J + 3, J + 2 and J + 1, and J + 1 has read it -- and keeps a barrier from running two
    // phases ahead of its waiter.
    auto receive = [&](uint32_t J, int j, float& m_prev) -> bool {
      if (J == 0) return true;
      const uint32_t pw = (uint32_t)(wg + 3) & 3u;
      if (!__all_sync(0xffffffffu, mbar_wait_flag(bars.at(Bars::kHand + 4 * pw + (warp & 3)), ((J - 1) / kSBufs) & 1, s_abort)))
        return false;
      if (j > 0) m_prev = s_hand[pw * 128 + row];
      return true;
    };

    FA4_FOR_EACH_TILE {
      const TileRec t = s_tiles[it];
      const int n = t.n;
      if (n <= 0) continue;
      float m_ref = kNegInf, l_sum = 0.f;

      for (int j = (wg - 2 * (int)gb) & 3; j < 2 * n; j += 4) {
        const uint32_t J = 2 * gb + j, slot = J % kPSlots;  // J % 4 == wg
        const int nb = kWindow ? window_visit_block(j >> 1, t) : (j >> 1);
        const int h64 = j & 1;
        const uint32_t bar_s = bars.at(Bars::kSFull + (wg & 2)), par_s = (J / kSBufs) & 1;

        // 1. the scores of this sub-block: the whole 64-key row of this thread
        ok = __all_sync(0xffffffffu, mbar_test(bar_s, par_s)) || __all_sync(0xffffffffu, mbar_wait_flag(bar_s, par_s, s_abort));
        if (!ok) break;
        tc_fence_after_sync();
        const bool cut = needs_mask<kWindow>(p, t, nb);     // some row of the tile does not see the whole block
        if constexpr (kWindow || kCache) {
          // None of the warp's 32 rows sees any of the 64 keys (the limits grow by one from row to row): P is zero, its
          // scales are the smallest, and the reference goes on as it came -- what the steps below would give.  A
          // quarter of the steps of a 127-key window, an eighth of those of a one-block causal tile.  us, masked -> left
          // out: 127-key window 75.4 -> 72.4; packed, 512 sequences of 128 242 -> 228, 64 of 512 175.0 -> 172.7, 4 of 8192
          // 1397 -> 1398; S = 8192, windows of 512, 1024, 4096 keys 152 -> 143, 229 -> 219, 576 -> 565; a chunk of 2048
          // against 32768 keys of a cache 746 -> 744.  Head dim 64 gains as much where tiles are short (143 -> 135, 217 -> 211;
          // 256 packed of 128 100.5 -> 98.0) and loses 0.5-0.9 % where they are long (window of 4096 552 -> 555, the
          // chunk 724 -> 728, 4 x 4096 through a cache 357 -> 359.5), one of 16384 keys 1.5 %.  (In the plain form, whose
          // tiles are long, the code costs more than it saves: causal GQA 1313 -> 1327.)
          const int r0 = (warp & 3) * 32;
          if (cut && (upper_key<kWindow>(p, t, r0 + 31, nb) < 64 * h64 ||
                      (kWindow && lower_key(p, t, r0, nb) > 64 * h64 + 63))) {
            mbar_arrive(bars.at(Bars::kSFree + wg));
            float m_prev = kNegInf;
            ok = receive(J, j, m_prev);
            if (!ok) break;
            s_hand[wg * 128 + row] = m_prev;
            mbar_arrive(bars.at(Bars::kHand + 4 * wg + (warp & 3)));
            if (m_prev != m_ref) l_sum *= reference_factor(m_ref, m_prev, sc.sl2);
            m_ref = m_prev;
            uint8_t* p_tile = gbase + kOffP + slot * kPTileBytes;
            *reinterpret_cast<uint4*>(p_tile + sw32_offset(row, 0)) = make_uint4(0u, 0u, 0u, 0u);
            *reinterpret_cast<uint4*>(p_tile + sw32_offset(row, 1)) = make_uint4(0u, 0u, 0u, 0u);
            *reinterpret_cast<uint32_t*>(gbase + kOffSFP + slot * 512 + (row & 31) * 16 + (row >> 5) * 4) = kMaskedScales;
            fence_proxy_async_smem();
            tc_fence_before_sync();
            mbar_arrive(bars.at(Bars::kPFull + slot));
            continue;
          }
        }
        if constexpr (!kNarrow) {
          if (cut) {
            if constexpr (kWindow) {
              ws::mask_scores_in_tmem_range(s_addr, lower_key(p, t, row, nb) - 64 * h64,
                                            upper_key<true>(p, t, row, nb) - 64 * h64);
            } else {
              mask_scores_in_tmem(s_addr, upper_key<false>(p, t, row, nb) - 64 * h64);
            }
          }
        }
        float s[64];
        tmem_ld32(s_addr, reinterpret_cast<uint32_t*>(&s[0]));
        tmem_ld32(s_addr + 32, reinterpret_cast<uint32_t*>(&s[32]));
        // While the scores travel (measured: 2.5 % of the kernel's time): the running reference.  Narrow windows take
        // it behind their maxima instead, below.
        float m_prev = kNegInf;
        if constexpr (!kNarrow) {
          if (J > 0) {
            const uint32_t pw = (uint32_t)(wg + 3) & 3u;
            ok = __all_sync(0xffffffffu, mbar_wait_flag(bars.at(Bars::kHand + 4 * pw + (warp & 3)), ((J - 1) / kSBufs) & 1, s_abort));
            if (!ok) break;
            if (j > 0) m_prev = s_hand[pw * 128 + row];
          }
        }
        tc_wait_ld();
        tc_fence_before_sync();
        mbar_arrive(bars.at(Bars::kSFree + wg));
        if constexpr (kNarrow) {
          if (cut)
            // (D = 192, whose registers are scarcer here, loses by the skip: 37.6 -> 38.1 us)
            mask_scores64<kD != 192>(s, lower_key(p, t, row, nb) - 64 * h64, upper_key<true>(p, t, row, nb) - 64 * h64,
                                     lower_key(p, t, (warp & 3) * 32 + 31, nb) - 64 * h64,
                                     upper_key<true>(p, t, (warp & 3) * 32, nb) - 64 * h64);
        }
        if constexpr (kCap) {
#pragma unroll
          for (int x = 0; x < 64; ++x) s[x] = soft_cap(s[x], sc.softcap_c1);
        }

        // 2. maxima of the four 16-key blocks, then the new reference
        if constexpr (kCutMax) {
          ok = code_boundary(slot + 2);
          if (!ok) break;
        }
        float bm4[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float m0 = fmax3(s[16 * q], s[16 * q + 1], s[16 * q + 2]);
          float m1 = fmax3(s[16 * q + 3], s[16 * q + 4], s[16 * q + 5]);
          m0 = fmax3(m0, s[16 * q + 6], s[16 * q + 7]);
          m1 = fmax3(m1, s[16 * q + 8], s[16 * q + 9]);
          m0 = fmax3(m0, s[16 * q + 10], s[16 * q + 11]);
          m1 = fmax3(m1, s[16 * q + 12], s[16 * q + 13]);
          m0 = fmax3(m0, s[16 * q + 14], s[16 * q + 15]);
          bm4[q] = fmaxf(m0, m1);
        }
        float m_loc = fmaxf(fmaxf(bm4[0], bm4[1]), fmaxf(bm4[2], bm4[3]));
        if constexpr (kNarrow) {
          // Masks and maxima take 800 clocks here, which four warps in a row would add up to the tile's time if each
          // began with the reference of the one before.  (The empty statement keeps the compiler from moving them
          // behind the wait.)  A long tile is better off with the two latencies beside each other.  us, reference first ->
          // maxima first: 127-key window 81 -> 75; causal GQA 1315 -> 1355.
          asm volatile("" : "+f"(m_loc), "+f"(bm4[0]), "+f"(bm4[1]), "+f"(bm4[2]), "+f"(bm4[3]));
          ok = receive(J, j, m_prev);
          if (!ok) break;
        }
        // (a seam for the compiler's scheduler here: 127-key window 90 -> 86.5 us, at D = 64 69.7 -> 69.0)
        if constexpr (kNarrow) __syncwarp();
        const float m_new = next_reference(m_prev, m_loc, sc.sl2);
        s_hand[wg * 128 + row] = m_new;
        mbar_arrive(bars.at(Bars::kHand + 4 * wg + (warp & 3)));
        auto follow_reference = [&] {            // own partial row sum
          if (m_new != m_ref) l_sum *= reference_factor(m_ref, m_new, sc.sl2);
          m_ref = m_new;
        };
        if constexpr (kSumFirst) follow_reference();
        float noff4[4];
        uint32_t sbits4[4], sf_bytes;
#if FA4_P_SCALE_E4M3
        block_scales4_e4m3(bm4, m_new, sc.sl2, noff4, sf_bytes, sbits4);
#else
        {
          uint32_t ue;
          block_exponents4(bm4, m_new, sc.sl2, noff4, ue);
          sf_bytes = block_scale_bytes(ue);
#pragma unroll
          for (int b4 = 0; b4 < 4; ++b4) sbits4[b4] = __byte_perm(ue, 0u, 0x4440u + b4) << 23;  // 2^e as fp32
        }
#endif
        if constexpr (!kSumFirst) follow_reference();

        // 3. exponentials and quantisation; P slot J % 8 is free: P V of sub-block J - 8 had run before these scores were made
        if constexpr (kCutExp) {
          ok = code_boundary(slot + 1);
          if (!ok) break;
        }
        uint8_t* p_tile = gbase + kOffP + slot * kPTileBytes;
        {
          uint32_t pk[8];
          float acc = 0.f;
#pragma unroll
          for (int b4 = 0; b4 < 4; ++b4) {
            const float bsum = quantize_block16(&s[16 * b4], noff4[b4], sc.sl2, pk[2 * b4], pk[2 * b4 + 1]);
            acc = fmaf(bsum, __uint_as_float(sbits4[b4]), acc);   // times the block scale
          }
          l_sum += acc;
          *reinterpret_cast<uint4*>(p_tile + sw32_offset(row, 0)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
          *reinterpret_cast<uint4*>(p_tile + sw32_offset(row, 1)) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
        }
        // the four scale bytes of this row: one word of the 512-byte chunk
        *reinterpret_cast<uint32_t*>(gbase + kOffSFP + slot * 512 + (row & 31) * 16 + (row >> 5) * 4) = sf_bytes;

        // 4. correction (rare, out of line): O holds the sub-blocks before this one relative to
        //    m_prev and must move to m_new before P V of this sub-block is issued; this thread
        //    owns its whole row of O
        //    (rows whose reference was -inf so far have an all-zero O: nothing to rescale)
        const bool fix = (m_new != m_prev) && (m_prev != kNegInf);
        if (j > 0 && __any_sync(0xffffffffu, fix)) {
          const uint32_t Jp = J - 1;
          ok = __all_sync(0xffffffffu, mbar_wait_flag(bars.at(Bars::kPvDone + (Jp % kPSlots)), (Jp / kPSlots) & 1, s_abort));
          if (!ok) break;
          tc_fence_after_sync();
          const float f = fix ? reference_factor(m_prev, m_new, sc.sl2) : 1.f;
          rescale_accumulator(lane_addr + o_column(ti), f, kDv / 32);
          tc_wait_st();
        }
        fence_proxy_async_smem();
        tc_fence_before_sync();
        mbar_arrive(bars.at(Bars::kPFull + slot));
      }
      if (!ok) break;

      // ---- tile end: hand the partial row sum and its reference to the epilogue warpgroup and
      //      go on with the next tile
      {
        const uint32_t fb = ti & 1;
        if (ti >= 2) {
          ok = __all_sync(0xffffffffu,
                          mbar_wait_flag(bars.at(Bars::kFinFree + fb), ((ti - 2) >> 1) & 1, s_abort));
          if (!ok) break;
        }
        volatile float* fin_slot = s_fin + fb * (4 * 128 * 2);
        // slot order = position of the warpgroup's first sub-block inside the tile: the summation
        // order of a row then depends on its tile only, not on what the CTA processed before
        const uint32_t fslot = (uint32_t)(wg - 2 * (int)gb) & 3u;
        fin_slot[(fslot * 128 + row) * 2] = l_sum;
        fin_slot[(fslot * 128 + row) * 2 + 1] = m_ref;
        mbar_arrive(bars.at(Bars::kFin + fb));
      }
      gb += n;
      ti += 1;
    }
  }
#undef FA4_FOR_EACH_TILE

  tc_fence_before_sync();
  __syncthreads();
  if (warp == kIssuerWarp) tmem_dealloc(tmem, kTmemCols);
}

}  // namespace fa4
