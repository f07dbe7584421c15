// Expert projections for more than one token on the tcgen05 tensor cores. One kernel takes every weight tile of a
// projection: the routed experts' (packed NVFP4 through tcgen05.mma.kind::mxf4nvf4.block_scale straight from the
// checkpoint layout, or BF16 banks through kind::f16) and the shared experts' (BF16). The weights are the M operand and
// stream from HBM; the tokens of an expert are the N operand.
//
// The N operand is laid out by a small kernel in front (`stage_rows_kernel`) exactly as the main kernel's ring wants it,
// tile by tile, so that the main kernel fetches it with one bulk copy per stage next to the weights and never gathers:
//   NVFP4  a token is four E2M1 digit rows with power-of-two block scales (tc_path.cuh); a tile is T = 16, 32 or 64 tokens;
//   BF16   a token is a row of 64-column pieces; a tile is 4 T tokens.
// (Gathering the digit rows in the main kernel, eight tokens a pass, stalled its MMAs at the head of every pass, and every
// expert's bank was read once per eight of its tokens: 64 tokens of one block 0.42 ms, 1 024 tokens 2.8 ms.)
//
// A ring stage is a chunk of the contraction (128 bytes of every row) of a tile of 128 weight rows and the N operand that goes
// with it: 8 stages of 27 KB, 6 of 36 KB or 4 of 54 KB. Prompts are bound by what crosses from L2 to the SMs: an image of 64 tokens is
// twice its weight tile's bytes, 8 GB in all for gate/up of 1 999 tokens at full width, 734 us = 10.9 TB/s (bulk copies alone reach 13.9).
// A larger T moves the weights less often, a smaller one leaves more of the ring to them: see gg_tokens.
//
// Persistent blocks, one per SM, that take the items from a counter (GgDeal). One warp deals, two produce, a stage each in turn (a stage's copies
// take the issuing lane 300 clocks), one thread issues the MMAs, four warps move block scales to tensor memory, four read accumulators and write outputs. The kernel is launched
// while its predecessor runs (programmatic dependent launch): until that is done it only streams weights, whose
// addresses depend on nothing but the plan. Every wait is bounded; one that gives up sets kFlagWaitTimedOut.
#include "../../include/inkling_b200.h"
#include "common.cuh"
#include "decode_args.cuh"
#include "mma_bf16.cuh"
#include "pipe.cuh"
#include "tc_path.cuh"
#include "tensor_map.cuh"

namespace ink {

// A stage: a tile of 128 rows x 128 B of weights, its block scales, the N operand, its block scales.
template <int T>
struct GgStage {
  static constexpr int kCount = T == 16 ? 8 : T == 32 ? 6 : 4;
  static constexpr int kScalesAt = kTcCodeBytes, kRowsAt = kScalesAt + kTcScaleBytes;
  static constexpr int kRowScalesAt = kRowsAt + T * 512, kBytes = (kRowScalesAt + T * 64 + 1023) / 1024 * 1024;
  static constexpr int kSf = T == 64 ? 48 : 32;   // tensor-memory columns of its scales
};
constexpr int kGgProducers = 2;
constexpr int kGgDealer = 10 + kGgProducers - 1;                  // the warp that deals the items out
constexpr int kGgThreads = (kGgDealer + 1) * 32;                 // (twelve warps: three on a scheduler, 168 registers a thread)
constexpr int kGgQueue = 8;                                      // items a block knows at once
constexpr int kGgDealStages = 16;                                // ring stages that a deal is worth at most
constexpr int kGgLateDeals = 4;                                  // deals that are left for a block after its first one, or more
constexpr int kGgMaxGroups = 1024;
constexpr int kGgPairRows = 16;                                  // shared experts: rows of gate and of up in turn
constexpr int kGgColD = 0, kGgColSf = 256;                       // tensor memory: two accumulators, then each stage's scales
constexpr int kGgAccCols = 128;                                  // of one: 32 tokens of digit rows or 128 BF16 tokens

// tokens in a tile
__host__ __device__ constexpr int gg_tile(bool fp4, int t) { return fp4 ? t : 4 * t; }
// slots of a group are padded to whole 1024-byte swizzle atoms of its tiles
__host__ __device__ constexpr int gg_pad(bool fp4) { return fp4 ? 2 : 8; }

struct GgArgs {
  // routed experts
  const unsigned char* maps;    // descriptors of this projection: codes and scales (NVFP4), or one (BF16)
  const int64_t* pointers;      // [(max_expert + 1) * stride]: a zero row is an inactive expert; scale2 is read through it
  const int32_t* experts;       // [groups]
  const int32_t* counts;        // [groups]
  const int32_t* rows;          // [groups, capacity]
  const unsigned char* image;   // N operand, group after group (see stage_rows_kernel)
  const unsigned char* image_scales;
  const float* slot_scale;      // [slots] (NVFP4)
  uint16_t* y;                  // BF16 [route][n / 2] (gate/up) or [route][n]
  int groups, start, capacity, stride, bank, k, n;
  // shared experts
  const unsigned char* shared_maps;    // gate and up in one, with a word behind it that says which comes first; or down
  const unsigned char* shared_image;   // [tile][k / 64][tokens of the tile, padded to 8][128 B]; down: the same per expert
  uint16_t* shared_y;           // gate/up: the image of the down projection; down: BF16 [tokens][n_shared][n]
  const uint16_t* gammas;       // [tokens, n_shared]
  int n_shared, tokens;
  unsigned* next;               // deals taken beyond the blocks' first ones; zero when this kernel's predecessor is done
  int32_t* status;
};

// One work item: a 128-row tile of one expert's matrix against one tile of its tokens.
struct GgItem {
  int shared;     // 1: of a shared expert; -1: no more items
  int group;      // group of routes, or shared expert
  int m0;         // first weight row
  int tile, n;    // tile of tokens, and how many
  int slot;       // first slot of the tile (routed)
};

struct GgShared {
  uint64_t full[8], empty[8], sf_full[8];
  uint64_t d_full[2], d_empty[2];
  uint64_t item_full[kGgQueue], item_empty[kGgQueue];
  GgItem items[kGgQueue];
  uint32_t tmem_base;
  volatile int taken;           // items the first producer has taken
  volatile int failed;
};

__device__ __forceinline__ bool gg_wait(uint64_t* bar, uint32_t parity, GgShared* sh) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (sh->failed) return false;
    if (clock64() - t0 > kWaitLimitCycles) {
      sh->failed = 1;
      return false;
    }
  }
  return true;
}

// routes of a group that have something to do
__device__ __forceinline__ int gg_count(const int32_t* counts, const int32_t* experts, const int64_t* pointers, int stride, int bank, int g) {
  const int count = counts[g], expert = experts[g];
  if (count <= 0 || expert < 0 || pointers[(size_t)expert * stride + bank] == 0) return 0;
  return count;
}

// Exclusive prefix sums of `mine` over a warp's lanes; *total gets the sum.
__device__ __forceinline__ int warp_before(int mine, int lane, int* total) {
  int up_to = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, up_to, o);
    if (lane >= o) up_to += v;
  }
  *total = __shfl_sync(0xffffffffu, up_to, 31);
  return up_to - mine;
}

// The groups' tables in shared memory: slot0[g] = first slot | padding slots of the group, before[g] = tiles (or routes) of
// all groups before. `slot0[g]` holds the group's count on entry.
struct GgTables { int* slot0; int* before; };
template <typename Of>
__device__ __forceinline__ void gg_scan(const GgTables& t, int groups, int pad, int lane, Of of) {
  int slots = 0, sum = 0;
  for (int g0 = 0; g0 < groups; g0 += 32) {
    const int g = g0 + lane, count = g < groups ? t.slot0[g] : 0;
    const int padded = (count + pad - 1) / pad * pad, c = of(count);
    int all_slots, all;
    const int s = slots + warp_before(padded, lane, &all_slots), w = sum + warp_before(c, lane, &all);
    if (g < groups) {
      t.slot0[g] = s | (padded - count);
      t.before[g] = w;
    }
    slots += all_slots;
    sum += all;
  }
  if (lane == 0) {
    t.slot0[groups] = slots;
    t.before[groups] = sum;
  }
}
// the group that holds number i of what `before` counts
__device__ __forceinline__ int gg_group_of(const int* before, int groups, int i) {
  int lo = 0, hi = groups;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (before[mid] <= i) lo = mid;
    else hi = mid;
  }
  return lo;
}
__device__ __forceinline__ int gg_first_slot(const int* slot0, int g, int pad) { return slot0[g] & ~(pad - 1); }
__device__ __forceinline__ int gg_group_count(const int* slot0, int g, int pad) {
  return gg_first_slot(slot0, g + 1, pad) - gg_first_slot(slot0, g, pad) - (slot0[g] & (pad - 1));
}

// The items in the order in which they are dealt: the shared experts' (the longest) first, then expert by expert the routed
// ones, all tiles of tokens of a tile of weight rows in a row. The blocks take them from one counter, a few ring stages'
// worth at a time, so that what runs at one time over the chip are the tiles of about five experts: the second tile of tokens of a weight
// tile finds the weights in L2, and so do the weight tiles of an expert the images of its tokens. (Dealt in contiguous shares
// by cost, each block read the weights again 0.8 MB later in its own stream, 120 MB over the chip, and two thirds of those
// reads went to DRAM: gate/up of 1 999 tokens at full width 985 us, now 734; down 490, now 410. No share is longer than another's:
// 61 tokens, gate/up 176 us, now 166, down 102, now 90; four tokens of a whole block 112, now 107.)
template <bool FP4, int T>
struct GgDeal {
  static constexpr int kTile = gg_tile(FP4, T), kPad = gg_pad(FP4), kSharedTile = gg_tile(false, T);
  const GgArgs* a;
  GgTables t;
  int m_tiles, shared_tiles;

  __device__ __forceinline__ int stages_of(bool shared) const { return a->k / ((FP4 && !shared) ? kTcChunkK : 64); }
  __device__ __forceinline__ int most_of(bool shared) const { return max(1, kGgDealStages / stages_of(shared)); }
  __device__ __forceinline__ int shared_items() const { return a->n_shared * m_tiles * shared_tiles; }
  __device__ __forceinline__ int routed_items() const { return t.before[a->groups] * m_tiles; }
  __device__ __forceinline__ GgItem shared_item(int i) const {
    GgItem it;
    const int per_e = m_tiles * shared_tiles;
    it.shared = 1;
    it.group = i / per_e;
    it.m0 = i % per_e / shared_tiles * kTcRows;
    it.tile = i % shared_tiles;
    it.n = min(kSharedTile, a->tokens - it.tile * kSharedTile);
    it.slot = 0;
    return it;
  }
  // routed item i; `group` is the group that holds it
  __device__ __forceinline__ GgItem routed_item(int i, int group) const {
    GgItem it;
    const int tiles = t.before[group + 1] - t.before[group], at = i - t.before[group] * m_tiles;
    const int first = gg_first_slot(t.slot0, group, kPad), count = gg_group_count(t.slot0, group, kPad);
    it.shared = 0;
    it.group = group;
    it.m0 = at / tiles * kTcRows;
    it.tile = at % tiles;
    it.n = min(kTile, count - it.tile * kTile);
    it.slot = first + it.tile * kTile;
    return it;
  }
};

// A role's way through the block's items: waits for the next one and takes it (whole warps call it).
struct GgTaker {
  uint32_t n = 0;
  __device__ __forceinline__ bool next(GgItem& it, GgShared* sh, int lane) {
    const uint32_t at = n % kGgQueue;
    const bool ok = __all_sync(0xffffffffu, gg_wait(&sh->item_full[at], n / kGgQueue & 1u, sh));
    if (!ok) return false;
    it = sh->items[at];
    __syncwarp();
    if (lane == 0) mbar_arrive(&sh->item_empty[at]);
    ++n;
    return it.shared >= 0;
  }
};

// E2M1 (block-scaled) items use tc_idesc; BF16 x BF16 -> FP32, M = 128:
__device__ __forceinline__ uint32_t gg_idesc_bf16(int n) { return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTcRows >> 4) << 24); }
// The four MMAs of a 128-byte chunk, from the low words of the operands' descriptors (tc_desc_sw128; the high word is the
// same for all, a step of 32 bytes adds 2). One block of instructions: the issuing thread is what a stage of few tokens waits
// for, and with descriptors put together one by one it took 80 (BF16) to 150 (block-scaled) clocks per MMA.
__device__ __forceinline__ uint32_t gg_desc_lo(uint32_t smem_addr) { return ((smem_addr >> 4) & 0x3fffu) | (1u << 16); }
constexpr uint32_t kGgDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ void gg_mma4_bf16(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p, q;\n .reg .b64 a, b;\n"
      " setp.ne.b32 p, %4, 0;\n setp.eq.b32 q, 0, 0;\n mov.b64 a, {%1, %5};\n mov.b64 b, {%2, %5};\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n add.s64 a, a, 2;\n add.s64 b, b, 2;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, q;\n add.s64 a, a, 2;\n add.s64 b, b, 2;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, q;\n add.s64 a, a, 2;\n add.s64 b, b, 2;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, q;\n}\n" ::"r"(d),
      "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(kGgDescHi)
      : "memory");
}
__device__ __forceinline__ void gg_mma4_fp4(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate, uint32_t sfa, uint32_t sfb) {
  asm volatile(
      "{\n .reg .pred p, q;\n .reg .b64 a, b;\n .reg .b32 s, t;\n"
      " setp.ne.b32 p, %4, 0;\n setp.eq.b32 q, 0, 0;\n mov.b64 a, {%1, %5};\n mov.b64 b, {%2, %5};\n mov.b32 s, %6;\n mov.b32 t, %7;\n"
      " tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], a, b, %3, [s], [t], p;\n"
      " add.s64 a, a, 2;\n add.s64 b, b, 2;\n add.s32 s, s, 4;\n add.s32 t, t, 4;\n"
      " tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], a, b, %3, [s], [t], q;\n"
      " add.s64 a, a, 2;\n add.s64 b, b, 2;\n add.s32 s, s, 4;\n add.s32 t, t, 4;\n"
      " tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], a, b, %3, [s], [t], q;\n"
      " add.s64 a, a, 2;\n add.s64 b, b, 2;\n add.s32 s, s, 4;\n add.s32 t, t, 4;\n"
      " tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], a, b, %3, [s], [t], q;\n}\n" ::"r"(d),
      "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(kGgDescHi), "r"(sfa), "r"(sfb)
      : "memory");
}
__device__ __forceinline__ bool elect_one() {
  uint32_t chosen;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(chosen));
  return chosen != 0;
}

template <bool FP4, int PROJ, int T>
__global__ void __launch_bounds__(kGgThreads, 1) grouped_gemm_kernel(const __grid_constant__ GgArgs a) {
  using Deal = GgDeal<FP4, T>;
  using St = GgStage<T>;
  // Two accumulators in turn: the next item's MMAs run while one is read. A tile of more than kGgAccCols columns (T = 64)
  // takes both. `acc` counts those a role has passed: number acc & 1, for the (acc >> 1)-th time.
  auto accs_of = [](const GgItem& it) -> int { return T < 64 ? 1 : it.n > (FP4 && !it.shared ? 32 : 128) ? 2 : 1; };
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ GgShared sh;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned char* ring = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // swizzled tiles: 1024-byte aligned
  GgTables tables;
  tables.slot0 = reinterpret_cast<int*>(ring + (size_t)St::kCount * St::kBytes);
  tables.before = tables.slot0 + a.groups + 1;
  Deal deal;
  deal.a = &a;
  deal.t = tables;
  deal.m_tiles = (a.n + kTcRows - 1) / kTcRows;
  deal.shared_tiles = a.n_shared > 0 ? (a.tokens + Deal::kSharedTile - 1) / Deal::kSharedTile : 0;

  for (int g = threadIdx.x; g < a.groups; g += kGgThreads) tables.slot0[g] = gg_count(a.counts, a.experts, a.pointers, a.stride, a.bank, g);
  if (threadIdx.x == 0) {
    for (int s = 0; s < St::kCount; ++s) {
      mbar_init(&sh.full[s], 1);
      mbar_init(&sh.empty[s], 1);
      mbar_init(&sh.sf_full[s], 4);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&sh.d_full[s], 1);
      mbar_init(&sh.d_empty[s], 4);
    }
    for (int s = 0; s < kGgQueue; ++s) {
      mbar_init(&sh.item_full[s], 1);
      mbar_init(&sh.item_empty[s], kGgProducers + 1 + (FP4 ? 4 : 0) + 4);   // every warp that takes items
    }
    sh.taken = 0;
    sh.failed = 0;
    mbar_init_fence();
  }
  if (warp == 1) tc_alloc(&sh.tmem_base, 512);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) gg_scan(tables, a.groups, Deal::kPad, lane, [](int count) { return (count + Deal::kTile - 1) / Deal::kTile; });
  __syncthreads();
  tc_fence_after();
  pdl_trigger();
  const uint32_t tmem = sh.tmem_base;

  if (warp == kGgDealer) {
    // =========================================================== the dealer
    // One lane. The first deal is the block's own number; the others come from the counter, which the kernel in front has
    // cleared, one deal ahead of the first producer: far enough to hide the counter's round trip (most deals last
    // longer), and no further, so that no block is left with items that others could have taken.
    if (lane == 0) {
      const int shared = deal.shared_items(), routed = deal.routed_items();
      // Items of a deal: at most sixteen stages' worth, and no more than leaves every block its part. A block's first deal is its share of the
      // items, as near as whole ones come, the later ones are a quarter of the share of what is left then. (Sixteen stages' worth throughout
      // left blocks without work in layers of short items: 1024 x 512, four choices, two tokens on 64 experts 35.4 us, 23.3 so; 75
      // tokens 45.5 / 39.7, 1 999 tokens 236 / 190, block of 1 499 tokens 245 / 200. A quarter of the items' share from the first deal on: 23.0,
      // 41.6, 196, 198; a half 23.0, 41.7, 217, 202. Long items, one or two a deal, are dealt as before: 1 999 tokens of 4096 x 2048 1 576 / 1 558.)
      const int blocks = (int)gridDim.x, per_s = min(deal.most_of(true), max(1, shared / blocks)), deals_s = (shared + per_s - 1) / per_s;
      const int most = deal.most_of(false), early_deals = max(0, blocks - deals_s);   // the blocks' first ones
      const int per_early = min(most, max(1, (routed + early_deals / 2) / max(1, early_deals))), left = max(0, routed - early_deals * per_early);
      const int per_late = min(most, max(1, left / (blocks * kGgLateDeals)));
      const int deals = deals_s + (left > 0 ? early_deals + (left + per_late - 1) / per_late : (routed + per_early - 1) / per_early);
      int dealt = 0;   // items dealt to this block
      auto put = [&](const GgItem& it) -> bool {
        const uint32_t at = (uint32_t)dealt % kGgQueue;
        if (dealt >= kGgQueue && !gg_wait(&sh.item_empty[at], (uint32_t)(dealt / kGgQueue - 1) & 1u, &sh)) return false;
        sh.items[at] = it;
        mbar_arrive(&sh.item_full[at]);
        ++dealt;
        return true;
      };
      bool ok = true, waited = false;
      for (int d = blockIdx.x; ok && d < deals;) {
        const int before = dealt;
        if (d < deals_s) {
          for (int i = d * per_s; ok && i < min(shared, (d + 1) * per_s); ++i) ok = put(deal.shared_item(i));
        } else {
          const int n = d - deals_s, late = n - early_deals, per = late < 0 ? per_early : per_late;
          const int first = late < 0 ? n * per_early : early_deals * per_early + late * per_late;
          int group = gg_group_of(tables.before, a.groups, first / deal.m_tiles);
          for (int i = first; ok && i < min(routed, first + per); ++i) {
            while (tables.before[group + 1] * deal.m_tiles <= i) ++group;
            ok = put(deal.routed_item(i, group));
          }
        }
        if (!waited) {
          pdl_wait();
          waited = true;
        }
        const long long t0 = clock64();
        while (ok && sh.taken <= before) {   // this deal's first item has not been taken
          if (sh.failed || clock64() - t0 > kWaitLimitCycles) {
            sh.failed = 1;
            ok = false;
          }
          __nanosleep(50);
        }
        d = (int)gridDim.x + (int)atomicAdd(a.next, 1u);
      }
      if (ok) {
        GgItem end = {};
        end.shared = -1;
        put(end);
      }
    }
    __syncwarp();
  } else if (warp == 0 || warp >= 10) {
    // =========================================================== producers
    const int producer = warp == 0 ? 0 : warp - 9;
    auto rows_bytes = [&](const GgItem& it) -> uint32_t {   // one chunk of the tile's N operand
      return (FP4 && !it.shared) ? (uint32_t)((it.n + 1) / 2 * 2) * 512u : (uint32_t)((it.n + 7) / 8 * 8) * 128u;
    };
    // (one elected lane issues a stage's copies one after the other: copies issued by several lanes of a warp at once were
    // taken apart lane by lane, 270 to 340 clocks each, 1 000 to 1 270 a stage)
    auto expect = [&](const GgItem& it, int u) {
      uint32_t bytes = kTcCodeBytes + rows_bytes(it);
      if (FP4 && !it.shared) bytes += kTcScaleBytes + rows_bytes(it) / 8u;
      mbar_expect_tx(&sh.full[u], bytes);
    };
    int bank = 0;   // index of the item's matrix
    auto issue_weights = [&](const GgItem& it, int s, int u) {
      unsigned char* stage = ring + (size_t)u * St::kBytes;
      uint64_t* bar = &sh.full[u];
      if (PROJ == 0 && it.shared) {   // gate and up rows, sixteen in turn: {column, row, which, block of rows, expert}
        tc_tma_5d(stage, a.shared_maps, s * 64, 0, 0, it.m0 / (2 * kGgPairRows), bank, bar);
      } else if (!FP4 || it.shared) {
        tc_tma_3d(stage, it.shared ? a.shared_maps : a.maps, s * 64, it.m0, bank, bar);
      } else {
        tc_tma_3d(stage, a.maps, s * 128, it.m0, bank, bar);
        tc_tma_3d(stage + St::kScalesAt, a.maps + 128, s * 16, it.m0, bank, bar);
      }
    };
    auto issue_rows = [&](const GgItem& it, int s, int u) {
      unsigned char* stage = ring + (size_t)u * St::kBytes;
      const uint32_t bytes = rows_bytes(it);
      const unsigned char* from;
      if (it.shared) {
        const int padded = (a.tokens + 7) / 8 * 8;
        from = a.shared_image + ((size_t)(PROJ ? it.group : 0) * padded + (size_t)it.tile * Deal::kSharedTile) * a.k * 2;
      } else {
        from = a.image + (size_t)it.slot * a.k * 2;
      }
      bulk_g2s(stage + St::kRowsAt, from + (size_t)s * bytes, bytes, &sh.full[u]);
      if (FP4 && !it.shared) bulk_g2s(stage + St::kRowScalesAt, a.image_scales + (size_t)it.slot * (a.k / 4) + (size_t)s * (bytes / 8), bytes / 8, &sh.full[u]);
    };
    // Stage i of the block's sequence is producer i % 2's. The first round's weights are asked for before the kernel in
    // front has finished; their N operand after.
    static_assert(St::kCount % kGgProducers == 0, "a ring slot has one producer");
    constexpr int kFirst = St::kCount / kGgProducers;   // stages of the first round per producer
    GgItem early_item[kFirst];
    int early_stage[kFirst], early = 0;
    GgItem it;
    long long first = 0;   // the block's stages before this item
    bool waited = false;
    auto rows_of_first_round = [&]() {
      pdl_wait();
      waited = true;
#pragma unroll
      for (int i = 0; i < kFirst; ++i)
        if (i < early && elect_one()) issue_rows(early_item[i], early_stage[i], producer + i * kGgProducers);
      __syncwarp();
    };
    GgTaker taker;
    while (true) {
      // (items beyond the queue's length arrive when others have taken theirs, which may wait for these rows)
      if (!waited && taker.n == kGgQueue) rows_of_first_round();
      if (!taker.next(it, &sh, lane)) break;
      if (producer == 0 && lane == 0) sh.taken = (int)taker.n;
      bank = it.shared ? it.group : a.experts[it.group] - a.start;
      const int stages = deal.stages_of(it.shared);
      int s = (int)((producer - first % kGgProducers + kGgProducers) % kGgProducers);
      for (; s < stages; s += kGgProducers) {
        const long long seq = first + s;
        const int u = (int)(seq % St::kCount);
        if (!waited && early < kFirst) {
          if (elect_one()) {
            expect(it, u);
            issue_weights(it, s, u);
          }
          __syncwarp();
#pragma unroll
          for (int i = 0; i < kFirst; ++i) {
            if (i == early) {
              early_item[i] = it;
              early_stage[i] = s;
            }
          }
          ++early;
          continue;
        }
        if (!waited) rows_of_first_round();
        if (seq >= St::kCount && !__all_sync(0xffffffffu, gg_wait(&sh.empty[u], (uint32_t)((seq / St::kCount) - 1) & 1u, &sh))) break;
        if (elect_one()) {
          expect(it, u);
          issue_weights(it, s, u);
          issue_rows(it, s, u);
        }
        __syncwarp();
      }
      first += stages;
      if (sh.failed) break;
    }
    if (!waited) rows_of_first_round();
  } else if (warp == 1) {
    // =========================================================== MMA issue
    // The whole warp walks the stages together (operands of the issue instructions are per-warp registers), one lane issues.
    GgItem it;
    uint32_t seq = 0;
    const uint32_t ring_lo = gg_desc_lo(smem_u32(ring));
    bool ok = true;
    GgTaker taker;
    for (uint32_t acc = 0; ok && taker.next(it, &sh, lane);) {
      const bool fp4 = FP4 && !it.shared;
      const int accs = __shfl_sync(0xffffffffu, accs_of(it), 0), n = __shfl_sync(0xffffffffu, it.n, 0);
      const int per_acc = fp4 ? 32 : 128, n_last = n - (accs - 1) * per_acc;
      auto idesc_of = [&](int tokens) { return fp4 ? tc_idesc((tokens + 1) / 2 * 8) : gg_idesc_bf16((tokens + 15) / 16 * 16); };
      const uint32_t idesc_last = idesc_of(n_last), idesc_first = accs > 1 ? idesc_of(per_acc) : idesc_last;
      const int stages = deal.stages_of(it.shared);
      const uint32_t d_first = tmem + kGgColD + (acc & 1) * kGgAccCols, d_second = tmem + kGgColD + ((acc + 1) & 1) * kGgAccCols;
      for (int i = 0; ok && i < accs; ++i) ok = gg_wait(&sh.d_empty[(acc + i) & 1], ((acc + i) >> 1 & 1u) ^ 1u, &sh);   // their previous items have been read
      if (!ok) break;
      tc_fence_after();
#pragma unroll 1
      for (int s = 0; s < stages; ++s, ++seq) {
        const uint32_t u = seq % St::kCount, parity = (seq / St::kCount) & 1u;
        ok = FP4 ? gg_wait(&sh.sf_full[u], parity, &sh) : gg_wait(&sh.full[u], parity, &sh);   // (the scales' warps have seen it full)
        if (FP4) ok = ok && gg_wait(&sh.full[u], parity, &sh);
        if (!ok) break;
        tc_fence_after();
        const uint32_t lo = ring_lo + u * (St::kBytes >> 4), rows = lo + (St::kRowsAt >> 4), sf = tmem + kGgColSf + u * St::kSf;
        if (elect_one()) {
          if (fp4) gg_mma4_fp4(d_first, lo, rows, idesc_first, s != 0, sf, sf + 16);
          else gg_mma4_bf16(d_first, lo, rows, idesc_first, s != 0);
          if (T == 64 && accs > 1) {   // the tile's upper half: 16 KB further in the N operand, whichever its type
            if (fp4) gg_mma4_fp4(d_second, lo, rows + (16384 >> 4), idesc_last, s != 0, sf, sf + 32);
            else gg_mma4_bf16(d_second, lo, rows + (16384 >> 4), idesc_last, s != 0);
          }
          tc_commit(&sh.empty[u]);
          if (s + 1 == stages) {
            tc_commit(&sh.d_full[acc & 1]);
            if (T == 64 && accs > 1) tc_commit(&sh.d_full[(acc + 1) & 1]);
          }
        }
        __syncwarp();
      }
      acc += accs;
    }
  } else if (warp < 6) {
    // =========================================================== block scales: shared -> tensor memory
    if constexpr (FP4) {
      const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;   // the tensor-memory subpartition this warp reaches
      GgItem it;
      long long seq = 0;
      bool ok = true;
      GgTaker taker;
      while (ok && taker.next(it, &sh, lane)) {
        const int stages = deal.stages_of(it.shared);
        for (int s = 0; s < stages; ++s, ++seq) {
          const int u = (int)(seq % St::kCount);
          ok = __all_sync(0xffffffffu, gg_wait(&sh.full[u], (uint32_t)(seq / St::kCount) & 1u, &sh));
          if (!ok) break;
          if (!it.shared) {
            const unsigned char* stage = ring + (size_t)u * St::kBytes;
            // row r's scales of a unit, 16 bytes, belong to lane r % 32, column r / 32, four bytes a 64-column step
            auto upload = [&](const unsigned char* sc, bool all, int column) {
              const uint4 r0 = *reinterpret_cast<const uint4*>(sc + lane * 16), r1 = *reinterpret_cast<const uint4*>(sc + (lane + 32) * 16);
              uint4 r2 = make_uint4(0, 0, 0, 0), r3 = r2;
              if (all) {
                r2 = *reinterpret_cast<const uint4*>(sc + (lane + 64) * 16);
                r3 = *reinterpret_cast<const uint4*>(sc + (lane + 96) * 16);
              }
              const uint32_t w[16] = {r0.x, r1.x, r2.x, r3.x, r0.y, r1.y, r2.y, r3.y, r0.z, r1.z, r2.z, r3.z, r0.w, r1.w, r2.w, r3.w};
              tc_st16(tmem + lane_base + kGgColSf + u * St::kSf + column, w);
            };
            tc_fence_after();
            upload(stage + St::kScalesAt, true, 0);
            upload(stage + St::kRowScalesAt, T > 16, 16);
            if (T == 64 && it.n > 32) upload(stage + St::kRowScalesAt + 2048, true, 32);
            tc_wait_st();
            tc_fence_before();
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh.sf_full[u]);
        }
      }
    }
  } else {
    // =========================================================== accumulators -> outputs
    pdl_wait();   // (the tokens' scales come from the kernel in front)
    const int sub = warp & 3;
    const uint32_t lane_base = (uint32_t)(sub * 32) << 16;
    GgItem it;
    bool ok = true;
    GgTaker taker;
    for (uint32_t acc = 0; ok && taker.next(it, &sh, lane);) {
      const bool fp4 = FP4 && !it.shared;
      const int expert = it.shared ? 0 : a.experts[it.group];
      const float scale2 = fp4 ? *reinterpret_cast<const float*>(a.pointers[(size_t)expert * a.stride + a.bank + 2]) : 1.f;
      const int per_chunk = fp4 ? 8 : 32, per_acc = fp4 ? 32 : 128;
      const int r = it.m0 + sub * 32 + lane;   // this thread's weight row
      // lane i holds token i of a chunk: its route (or token number), and its scale
      auto token_of = [&](int at, float& scale) -> int {   // `at`: the chunk's first token in the tile
        const int i = at + lane;
        scale = 0.f;
        if (lane >= per_chunk || i >= it.n) return -1;
        if (it.shared) return it.tile * Deal::kSharedTile + i;
        if (fp4) scale = scale2 * a.slot_scale[it.slot + i];
        return a.rows[(size_t)it.group * a.capacity + it.tile * Deal::kTile + i];
      };
      // this thread's weight row for the tokens at .. of a chunk (lane j holds token j's route, or number)
      auto write = [&](auto& v, int at, int tokens) {
        constexpr int kChunk = sizeof(v) / sizeof(float);
        const int here = min(kChunk, it.n - at);
        if (PROJ == 0) {
          // gate and up rows alternate, so neighbouring lanes hold a pair: of two tokens each lane finishes one
          const bool second = (lane & 1) != 0;
          const int pair = r >> 1;
#pragma unroll
          for (int j = 0; j < kChunk; j += 2) {
            if (j >= here) break;
            const float other = __shfl_xor_sync(0xffffffffu, second ? v[j] : v[j + 1], 1);
            const float gate = second ? other : v[j], up = second ? v[j + 1] : other;
            const int token = __shfl_sync(0xffffffffu, tokens, second ? j + 1 : j);
            if (token >= 0) a.y[(size_t)token * (a.n / 2) + pair] = (uint16_t)f32_to_bf16_bits(silu_mul(gate, up));
          }
        } else {
#pragma unroll
          for (int j = 0; j < kChunk; ++j) {
            if (j >= here) break;
            const int token = __shfl_sync(0xffffffffu, tokens, j);
            uint16_t* y = it.shared ? a.shared_y + ((size_t)token * a.n_shared + it.group) * a.n : a.y + (size_t)token * a.n;
            y[r] = (uint16_t)f32_to_bf16_bits(v[j]);
          }
        }
      };
      if constexpr (FP4) {
        if (!it.shared) {
          // Everything into registers first (four digit columns add up to a token), so that the accumulators are free for the
          // next items before the outputs are written: written one by one, the second waited for the first one's outputs and
          // the MMAs for both (a fifth of the gate/up projection of 1 999 tokens).
          constexpr int kChunks = T / 8;
          float v[kChunks][8], my_scale;
          int my_token = token_of(0, my_scale);   // (asked for before the wait)
#pragma unroll
          for (int i = 0; i < (T == 64 ? 2 : 1); ++i) {
            if (i * 32 >= it.n) break;
            const int buf = acc & 1;
            ok = __all_sync(0xffffffffu, gg_wait(&sh.d_full[buf], (acc >> 1) & 1u, &sh));
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < (T < 32 ? T : 32) / 8; ++c) {
              if (i * 32 + c * 8 >= it.n) break;
              float w[32];
              tc_ld32(tmem + lane_base + kGgColD + buf * kGgAccCols + c * 32, w);
#pragma unroll
              for (int j = 0; j < 8; ++j) v[i * 4 + c][j] = (w[4 * j] + w[4 * j + 1]) + (w[4 * j + 2] + w[4 * j + 3]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.d_empty[buf]);
            ++acc;
          }
          if (!ok) break;
#pragma unroll
          for (int chunk = 0; chunk < kChunks; ++chunk) {
            if (chunk * 8 >= it.n) break;
            if (chunk > 0) my_token = token_of(chunk * 8, my_scale);
#pragma unroll
            for (int j = 0; j < 8; ++j) v[chunk][j] *= __shfl_sync(0xffffffffu, my_scale, j);
            write(v[chunk], chunk * 8, my_token);
          }
          continue;
        }
      }
#pragma unroll 1
      for (int first = 0; first < it.n; first += per_acc, ++acc) {   // (an item's accumulators, one after the other)
        const int buf = acc & 1, here_n = min(per_acc, it.n - first), token_chunks = (here_n + per_chunk - 1) / per_chunk;
        const uint32_t d = tmem + lane_base + kGgColD + buf * kGgAccCols;
        float unused;
        const int first_token = token_of(first, unused);
        ok = __all_sync(0xffffffffu, gg_wait(&sh.d_full[buf], (acc >> 1) & 1u, &sh));
        if (!ok) break;
        tc_fence_after();
        if (PROJ == 0 && it.shared) {
          // lanes 0-15 hold sixteen pairs' gate rows, lanes 16-31 their up rows (or the other way round): of two tokens each
          // lane finishes one
          const bool second = (lane & 16) != 0, up_first = *reinterpret_cast<const int*>(a.shared_maps + 128) != 0;
          const int pair = it.m0 / 2 + sub * kGgPairRows + (lane & 15), padded = (a.tokens + 7) / 8 * 8, f = a.n / 2;
          unsigned char* tile = reinterpret_cast<unsigned char*>(a.shared_y) + ((size_t)it.group * padded + (size_t)it.tile * Deal::kSharedTile) * f * 2 +
                                (size_t)(pair >> 6) * ((it.n + 7) / 8 * 8) * 128 + (pair & 7) * 2;
#pragma unroll 1
          for (int chunk = 0; chunk < token_chunks; ++chunk) {
            float v[32];
            tc_ld32(d + chunk * 32, v);
            const int here = min(32, here_n - chunk * 32);
            const int at0 = first + chunk * 32, mine = min(at0 + lane, it.n - 1);   // (lane j's gamma is that of token j)
            const float my_gamma = bf16_to_f32(a.gammas[(size_t)(it.tile * Deal::kSharedTile + mine) * a.n_shared + it.group]);
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
              if (j >= here) break;
              // the reference's BF16 tensor ops: both bmm outputs, silu, the product and the product with gamma round
              const float other = __shfl_xor_sync(0xffffffffu, second ? v[j] : v[j + 1], 16), own = second ? v[j + 1] : v[j];
              const float gamma = __shfl_sync(0xffffffffu, my_gamma, second ? j + 1 : j);
              const float g = round_bf16(second != up_first ? other : own), u = round_bf16(second != up_first ? own : other);
              const float act = round_bf16(round_bf16(g / (1.f + expf(-g))) * u);
              const int at = at0 + j + (second ? 1 : 0);
              if (at < it.n) *reinterpret_cast<uint16_t*>(tile + at * 128 + ((((pair & 63) >> 3) ^ (at & 7)) << 4)) = (uint16_t)f32_to_bf16_bits(act * gamma);
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh.d_empty[buf]);
          continue;
        }
        if constexpr (!FP4 || PROJ == 1) {
#pragma unroll 1
          for (int chunk = 0; chunk < token_chunks; ++chunk) {
            const int tokens = chunk > 0 ? token_of(first + chunk * 32, unused) : first_token;
            float v[32];
            tc_ld32(d + chunk * 32, v);
            write(v, first + chunk * 32, tokens);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.d_empty[buf]);
      }
    }
  }
  __syncwarp();
  pdl_wait();   // whoever waits for this kernel may rely on the ones before it too
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tc_dealloc(tmem, 512);
  if (threadIdx.x == 0 && sh.failed && a.status) atomicOr(a.status, kFlagWaitTimedOut);
}

// ---------------------------------------------------------------------------- N operand
struct StageArgs {
  const uint16_t* x;            // BF16 [*, k]
  const int64_t* pointers;
  const int32_t *experts, *counts, *rows;
  unsigned char* image;         // routed slots; a tile of n tokens: [chunk][n padded][4 digit rows x 128 B] or [chunk][n padded][128 B]
  unsigned char* image_scales;  // NVFP4: [chunk][n padded][4 digit rows x 16 B] per tile
  float* slot_scale;
  unsigned char* shared_image;  // the tokens themselves for the shared experts, or null
  int groups, capacity, stride, bank, k, div;   // div: routes per row of x
  int plan_ready;               // the plan was complete before the kernel in front started
  unsigned* next;               // the main kernel's counter of deals, cleared here
  int tokens, tile, shared_tile;
};

constexpr int kStageThreads = 128;

// 16-byte pieces of a BF16 row into a [k / 64][rows][128 B] swizzled image
__device__ __forceinline__ void stage_bf16_row(const uint16_t* from, unsigned char* tile, int row, int padded, int k) {
  for (int p = threadIdx.x; p < k / 8; p += kStageThreads)
    *reinterpret_cast<uint4*>(tile + (size_t)(p >> 3) * padded * 128 + row * 128 + (((p & 7) ^ (row & 7)) << 4)) = reinterpret_cast<const uint4*>(from)[p];
}

// Blocks take routed slots in turn, then the tokens for the shared experts. Bound by the digit arithmetic (tc_digits8; more
// blocks an SM, 12 or 16 for 8, changed nothing) and, for prompts, by the image's bytes; a token is converted once per route, which
// costs less than gathering it from one copy sixteen times per expert in the main kernel.
template <bool FP4>
__global__ void __launch_bounds__(kStageThreads) stage_rows_kernel(StageArgs a) {
  extern __shared__ __align__(16) int s_tables[];
  __shared__ uint32_t s_amax[kStageThreads / 32];
  constexpr int kPad = gg_pad(FP4);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  GgTables t{s_tables, s_tables + a.groups + 1};
  if (!a.plan_ready) {
    pdl_wait();
    pdl_trigger();   // the main kernel may read the plan now
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.next = 0;   // (nothing in flight uses it: each projection of a call has its own)
  for (int g = threadIdx.x; g < a.groups; g += kStageThreads) t.slot0[g] = gg_count(a.counts, a.experts, a.pointers, a.stride, a.bank, g);
  __syncthreads();
  if (warp == 0) gg_scan(t, a.groups, kPad, lane, [](int count) { return count; });
  __syncthreads();
  const int routed = t.before[a.groups], total = routed + (a.shared_image ? a.tokens : 0);
  if (a.plan_ready) {
    pdl_wait();
    pdl_trigger();
  }
  for (int i = blockIdx.x; i < total; i += gridDim.x) {
    if (i >= routed) {
      const int token = i - routed, tile = token / a.shared_tile, row = token % a.shared_tile;
      const int padded = (min(a.shared_tile, a.tokens - tile * a.shared_tile) + 7) / 8 * 8;
      stage_bf16_row(a.x + (size_t)token * a.k, a.shared_image + (size_t)tile * a.shared_tile * a.k * 2, row, padded, a.k);
      continue;
    }
    const int lo = gg_group_of(t.before, a.groups, i);   // the group of active route i
    const int pos = i - t.before[lo], count = t.before[lo + 1] - t.before[lo];
    const int tile = pos / a.tile, row = pos % a.tile, slot0 = gg_first_slot(t.slot0, lo, kPad) + tile * a.tile;
    const int padded = (min(a.tile, count - tile * a.tile) + kPad - 1) / kPad * kPad;
    const uint16_t* from = a.x + (size_t)(a.rows[(size_t)lo * a.capacity + pos] / a.div) * a.k;
    if constexpr (!FP4) {
      stage_bf16_row(from, a.image + (size_t)slot0 * a.k * 2, row, padded, a.k);
    } else {
      const uint4* x = reinterpret_cast<const uint4*>(from);
      constexpr int kMost = kTcMaxK / 8 / kStageThreads;
      uint4 v[kMost];
      uint32_t amax = 0;
#pragma unroll
      for (int n = 0; n < kMost; ++n) {
        const int p = n * kStageThreads + threadIdx.x;
        v[n] = p < a.k / 8 ? x[p] : make_uint4(0, 0, 0, 0);
        const uint32_t w4[4] = {v[n].x, v[n].y, v[n].z, v[n].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) amax = max(amax, max(w4[j] & 0x7fffu, (w4[j] >> 16) & 0x7fffu));
      }
      amax = __reduce_max_sync(0xffffffffu, amax);
      __syncthreads();   // (the previous slot's maxima have been read)
      if (lane == 0) s_amax[warp] = amax;
      __syncthreads();
#pragma unroll
      for (int w = 0; w < kStageThreads / 32; ++w) amax = max(amax, s_amax[w]);
      float inverse;
      const float scale = pow2_normaliser(amax, &inverse);
      const float below = amax >= 0x7f00u ? 256.f : 512.f;   // brings the largest below 1024 (2^127 and more: normalised to [2, 4))
      // (digits cannot hold a NaN or an infinity: the token's scale carries it into all of its results)
      if (threadIdx.x == 0) a.slot_scale[slot0 + row] = amax >= 0x7f80u ? __int_as_float(0x7fffffff) : inverse / below;
      unsigned char* image = a.image + (size_t)slot0 * a.k * 2 + (size_t)row * 512;
      unsigned char* scales = a.image_scales + (size_t)slot0 * (a.k / 4) + (size_t)row * 64;
#pragma unroll
      for (int n = 0; n < kMost; ++n) {
        const int p = n * kStageThreads + threadIdx.x, chunk = p >> 5;   // a warp holds a chunk of 256 elements
        if (chunk * kTcChunkK < a.k)
          tc_stage8_row(v[n], below * scale, image + (size_t)chunk * padded * 512, 4 * (row & 1), scales + (size_t)chunk * padded * 64, lane);
      }
    }
  }
}

// ---------------------------------------------------------------------------- combine
// out[token] = sum over choices of fp32(bf16(y[route] * w)) in choice order, then the shared experts: eight columns a thread
__global__ void __launch_bounds__(256) combine_kernel(const uint16_t* __restrict__ y, const int64_t* __restrict__ indices,
                                                      const uint16_t* __restrict__ weights, const int64_t* __restrict__ pointers, int stride, int max_expert,
                                                      const uint16_t* __restrict__ shared_y, int n_shared, float* out, uint16_t* out_bf16,
                                                      int width, int top_k, int32_t* status) {
  pdl_wait();
  pdl_trigger();
  const int token = blockIdx.x, piece = blockIdx.y * 256 + threadIdx.x;
  if (piece * 8 >= width) return;
  float sum[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) sum[i] = 0.f;
  for (int j = 0; j < top_k; ++j) {
    const size_t route = (size_t)token * top_k + j;
    const int64_t expert = indices[route];
    if (expert < 0 || expert > max_expert) {
      if (piece == 0 && status) atomicOr(status, kFlagExpertOutOfRange);
      continue;
    }
    if (pointers[expert * stride] == 0) continue;
    const float w = bf16_to_f32(weights[route]);
    const uint4 q = __ldcg(reinterpret_cast<const uint4*>(y + route * width) + piece);   // (y is written while this kernel is on the chip)
    const uint32_t q4[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      sum[2 * i] += round_bf16(bf16lo(q4[i]) * w);
      sum[2 * i + 1] += round_bf16(bf16hi(q4[i]) * w);
    }
  }
  for (int e = 0; e < n_shared; ++e) {
    const uint4 q = __ldcg(reinterpret_cast<const uint4*>(shared_y + ((size_t)token * n_shared + e) * width) + piece);
    const uint32_t q4[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      sum[2 * i] += bf16lo(q4[i]);
      sum[2 * i + 1] += bf16hi(q4[i]);
    }
  }
  if (out) {
    float4* to = reinterpret_cast<float4*>(out + (size_t)token * width) + 2 * piece;
    to[0] = make_float4(sum[0], sum[1], sum[2], sum[3]);
    to[1] = make_float4(sum[4], sum[5], sum[6], sum[7]);
  }
  if (out_bf16) {
    uint4 p;
    p.x = f32_to_bf16_bits(sum[0]) | (f32_to_bf16_bits(sum[1]) << 16);
    p.y = f32_to_bf16_bits(sum[2]) | (f32_to_bf16_bits(sum[3]) << 16);
    p.z = f32_to_bf16_bits(sum[4]) | (f32_to_bf16_bits(sum[5]) << 16);
    p.w = f32_to_bf16_bits(sum[6]) | (f32_to_bf16_bits(sum[7]) << 16);
    reinterpret_cast<uint4*>(out_bf16 + (size_t)token * width)[piece] = p;
  }
}

// ---------------------------------------------------------------------------- host side
static size_t gg_pad256(size_t n) { return (n + 255) / 256 * 256; }

// what one projection's N operand takes: images of the routed slots, of the tokens for the shared experts
struct GgScratch {
  size_t slots, image, image_scales, slot_scale, next, total;
  GgScratch(bool fp4, size_t routes, size_t groups, int k) {
    const size_t active = routes < groups ? routes : groups;
    slots = routes + active * (gg_pad(fp4) - 1);
    image = gg_pad256(slots * (size_t)k * 2);
    image_scales = fp4 ? gg_pad256(slots * (size_t)k / 4) : 0;
    slot_scale = fp4 ? gg_pad256(slots * sizeof(float)) : 0;
    next = 256;   // the counter of deals
    total = image + image_scales + slot_scale + next;
  }
};

static int gg_sms() {
  constexpr int kMaxDevices = 64;
  static int sms_of[kMaxDevices] = {};
  int device = 0;
  cudaGetDevice(&device);
  if (device < 0 || device >= kMaxDevices) return 148;
  if (sms_of[device] == 0) {
    int count = 0;
    cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device);
    sms_of[device] = count < 1 ? 148 : count;
  }
  return sms_of[device];
}

// launched while the kernel in front runs (both sides use griddepcontrol)
template <typename Args>
static cudaError_t launch_dependent(void (*kernel)(Args), dim3 grid, int threads, size_t smem, cudaStream_t stream, const Args& args) {
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = dim3(threads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attribute;
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  config.attrs = &attribute;
  config.numAttrs = 1;
  return cudaLaunchKernelEx(&config, kernel, args);
}

template <bool FP4, int PROJ, int T>
static int launch_grouped(const GgArgs& a, cudaStream_t stream) {
  constexpr size_t kRing = (size_t)GgStage<T>::kCount * GgStage<T>::kBytes + 1024;
  static_assert(kGgColSf + GgStage<T>::kCount * GgStage<T>::kSf <= 512, "tensor memory");
  constexpr int kMaxDevices = 64;
  static bool configured[kMaxDevices] = {};
  int device = 0;
  cudaGetDevice(&device);
  INK_REQUIRE(device >= 0 && device < kMaxDevices, kLaunchFailed, "grouped projections: device ordinal %d", device);
  if (!configured[device]) {
    constexpr size_t most = kRing + 2 * sizeof(int) * (kGgMaxGroups + 1);
    static_assert(most + sizeof(GgShared) <= 227 * 1024, "shared memory");
    cudaError_t e = cudaFuncSetAttribute(grouped_gemm_kernel<FP4, PROJ, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    INK_REQUIRE(e == cudaSuccess, kLaunchFailed, "grouped projections: %zu bytes of shared memory refused: %s", most, cudaGetErrorString(e));
    configured[device] = true;
  }
  const cudaError_t e = launch_dependent(grouped_gemm_kernel<FP4, PROJ, T>, dim3(gg_sms()), kGgThreads,
                                         kRing + 2 * sizeof(int) * (a.groups + 1), stream, a);
  INK_REQUIRE(e == cudaSuccess, kLaunchFailed, "grouped projections: launch failed: %s", cudaGetErrorString(e));
  return kOk;
}
template <bool FP4, int PROJ>
static int launch_grouped(int tokens, const GgArgs& a, cudaStream_t s) {
  return tokens == 64 ? launch_grouped<FP4, PROJ, 64>(a, s) : tokens == 32 ? launch_grouped<FP4, PROJ, 32>(a, s) : launch_grouped<FP4, PROJ, 16>(a, s);
}

static int launch_stage(bool fp4, const StageArgs& a, size_t most_rows, cudaStream_t stream) {
  const size_t smem = 2 * sizeof(int) * (a.groups + 1), most = (size_t)gg_sms() * 8;
  const dim3 grid((unsigned)(most_rows < most ? most_rows : most));
  const cudaError_t e = fp4 ? launch_dependent(stage_rows_kernel<true>, grid, kStageThreads, smem, stream, a)
                            : launch_dependent(stage_rows_kernel<false>, grid, kStageThreads, smem, stream, a);
  INK_REQUIRE(e == cudaSuccess, kLaunchFailed, "grouped projections: launch failed: %s", cudaGetErrorString(e));
  return kOk;
}

// Tokens T of a tile, from the mean number of routes per expert. T = 16, 32, 64, us a call, experts chosen evenly / as rank^-0.6:
//   256 of 4096 x 2048   mean 8: 580 597 652 / 603 604 652;  16:  713 646 707 /  748  678  725;  32: 1181  873  849 / 1225  920  890;  48: 1608 1232 1006 / 1594 1121 1061
//   256 of 4096 x 512         8: 222 225 237 / 224 228 257;  16:  292 280 289 /  295  293  312;  32:  486  418  417 /  489  423  441;  48:  694  583  553 /  701  581  576
//   128 of 2048 x 1024        8: 111 109 116 / 114 117 128;  16:  137 128 132 /  141  138  155;  32:  220  195  184 /  221  188  194;  48:  302  258  247 /  294  254  261
//    64 of 1024 x 512         8:  42  42  41 /  44  48  47;  16:   51  50  50 /   51   54   70;  32:   71   70   71 /   73   71   85;  48:   94   91   92 /   94   93  100
// T = 16 and 32 meet between means of 10 (595 609 / 639 622 for the largest layers) and 12 (618 622 / 676 640). The lines are those of long items: where
// items are short and the choice uneven a smaller tile would do better, by up to 12 % (the last row, means of 12, 16, 40 and 48).
static int gg_tokens(long long routes, int experts) { return routes > 32LL * experts ? 64 : routes > 10LL * experts ? 32 : 16; }

}  // namespace ink

using namespace ink;

extern "C" int ink_encode_bf16_banks(void* out_host_256, const void* gate_up, uint64_t gate_up_stride, const void* down, uint64_t down_stride,
                                     int experts, int hidden, int intermediate) {
  INK_REQUIRE(out_host_256 != nullptr && experts >= 1, kBadArgument, "encode_bf16_banks: null output or no experts");
  INK_REQUIRE(hidden % 64 == 0 && intermediate % 64 == 0, kUnsupportedShape, "encode_bf16_banks: hidden=%d intermediate=%d", hidden, intermediate);
  CUtensorMap maps[2];
  int rc = encode_rows(&maps[0], gate_up, 2, gate_up_stride, experts, 2 * intermediate, hidden, 64, kTcRows, true);
  if (rc == kOk) rc = encode_rows(&maps[1], down, 2, down_stride, experts, hidden, intermediate, 64, kTcRows, true);
  if (rc == kOk) memcpy(out_host_256, maps, sizeof(maps));
  return rc;
}

extern "C" int ink_encode_shared(void* out_host_384, const void* gate, const void* up, const void* down, int n_shared, int hidden, int intermediate) {
  INK_REQUIRE(out_host_384 != nullptr && n_shared >= 1, kBadArgument, "encode_shared: null output or no experts");
  INK_REQUIRE(hidden % 64 == 0 && intermediate % 64 == 0, kUnsupportedShape, "encode_shared: hidden=%d intermediate=%d", hidden, intermediate);
  // Gate and up in one descriptor, sixteen rows of each in turn, the one at the lower address first; the word
  // that follows it is not zero if that is `up`.
  const bool up_first = (uintptr_t)up < (uintptr_t)gate;
  const uintptr_t low = (uintptr_t)(up_first ? up : gate), high = (uintptr_t)(up_first ? gate : up);
  const uint64_t stride = 2ull * hidden * intermediate, row_bytes = 2ull * hidden;
  unsigned char maps[384] = {};
  TensorMapEncodeFn enc = tensor_map_encoder();
  INK_REQUIRE(enc != nullptr, kLaunchFailed, "encode_shared: the driver has no cuTensorMapEncodeTiled");
  INK_REQUIRE(low != 0 && low % 16 == 0 && high % 16 == 0 && high > low && high - low < (1ull << 40), kMisaligned,
              "encode_shared: gate at %p and up at %p", gate, up);
  cuuint64_t dims[5] = {(cuuint64_t)hidden, (cuuint64_t)kGgPairRows, 2, (cuuint64_t)(intermediate / kGgPairRows), (cuuint64_t)n_shared};
  cuuint64_t strides[4] = {row_bytes, high - low, kGgPairRows * row_bytes, stride};
  cuuint32_t box[5] = {64, (cuuint32_t)kGgPairRows, 2, (cuuint32_t)(kTcRows / 2 / kGgPairRows), 1}, elem[5] = {1, 1, 1, 1, 1};
  CUtensorMap both;
  const CUresult r = enc(&both, CU_TENSOR_MAP_DATA_TYPE_UINT16, 5, (void*)low, dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  INK_REQUIRE(r == CUDA_SUCCESS, kBadArgument, "encode_shared: cuTensorMapEncodeTiled returned %d", (int)r);
  memcpy(maps, &both, sizeof(both));
  maps[128] = up_first ? 1 : 0;
  CUtensorMap last;
  if (int rc = encode_rows(&last, down, 2, stride, n_shared, hidden, intermediate, 64, kTcRows, true)) return rc;
  memcpy(maps + 256, &last, sizeof(last));
  memcpy(out_host_384, maps, sizeof(maps));
  return kOk;
}

// The items are counted in 32 bits, with room to spare: 16 million routes at the greatest widths.
static int check_items_fit(bool fp4, size_t routes, int groups, int n, int t) {
  const size_t tiles = routes / gg_tile(fp4, t) + (size_t)groups;
  INK_REQUIRE(tiles * (n / kTcRows) * 128 <= 0x7fffffff && routes <= 0x40000000, kUnsupportedShape,
              "grouped projections: %zu routes in one call", routes);
  return kOk;
}

static int check_grouped_shape(bool fp4, int n, int k, int groups) {
  const int step = fp4 ? kTcChunkK : 64;
  INK_REQUIRE(k % step == 0 && k >= step && k <= kTcMaxK && n % kTcRows == 0 && n > 0, kUnsupportedShape,
              "grouped projections: n=%d k=%d unsupported (n a multiple of %d, k a multiple of %d up to %d)", n, k, kTcRows, step, kTcMaxK);
  INK_REQUIRE(groups >= 0 && groups <= kGgMaxGroups, kBadArgument, "grouped projections: %d groups, at most %d", groups, kGgMaxGroups);
  return kOk;
}

extern "C" size_t ink_moe_grouped_scratch_bytes(int tokens, int top_k, int n_shared, int hidden, int intermediate, int groups, int quantized) {
  const size_t routes = (size_t)(tokens > 0 ? tokens : 0) * top_k, padded = ((size_t)(tokens > 0 ? tokens : 0) + 7) / 8 * 8;
  const GgScratch a(quantized != 0, routes, groups, hidden), b(quantized != 0, routes, groups, intermediate);
  return a.total + b.total + gg_pad256(n_shared ? padded * hidden * 2 : 0) + gg_pad256(padded * n_shared * intermediate * 2) +
         gg_pad256((size_t)(tokens > 0 ? tokens : 0) * n_shared * hidden * 2);
}

extern "C" int ink_moe_grouped(const void* x, const int64_t* indices, const void* weights, const int64_t* pointers, const int32_t* experts,
                               const int32_t* rows, const int32_t* counts, const void* bank_maps, const void* shared_maps, const void* gammas,
                               void* activated, void* down, float* output, void* output_bf16, int tokens, int top_k, int n_shared, int hidden, int intermediate, int groups,
                               int start, int local, int capacity, int max_expert, int quantized, void* scratch, size_t scratch_bytes, int32_t* status,
                               ink_stream_t stream) {
  INK_REQUIRE(x && indices && weights && pointers && experts && rows && counts && bank_maps && activated && down && scratch && (output || output_bf16), kBadArgument,
              "moe_grouped: null pointer argument");
  INK_REQUIRE(n_shared == 0 || (shared_maps && gammas), kBadArgument, "moe_grouped: shared experts need their descriptors and weights");
  INK_REQUIRE(tokens >= 0 && top_k >= 1 && n_shared >= 0 && capacity >= 1 && start >= 0 && local >= 1, kBadArgument,
              "moe_grouped: tokens=%d top_k=%d n_shared=%d capacity=%d", tokens, top_k, n_shared, capacity);
  const bool fp4 = quantized != 0;
  if (int rc = check_grouped_shape(fp4, 2 * intermediate, hidden, groups)) return rc;
  if (int rc = check_grouped_shape(fp4, hidden, intermediate, groups)) return rc;
  const size_t routes = (size_t)tokens * top_k, padded = ((size_t)tokens + 7) / 8 * 8;
  const int t = gg_tokens((long long)routes, local);
  if (int rc = check_items_fit(fp4, routes, groups, 2 * intermediate > hidden ? 2 * intermediate : hidden, t)) return rc;
  INK_REQUIRE(scratch_bytes >= ink_moe_grouped_scratch_bytes(tokens, top_k, n_shared, hidden, intermediate, groups, quantized), kBadArgument,
              "moe_grouped: scratch of %zu bytes is too small", scratch_bytes);
  INK_REQUIRE(aligned16(x) && aligned16(activated) && aligned16(down) && aligned16(output) && aligned16(output_bf16) && (reinterpret_cast<uintptr_t>(scratch) & 255u) == 0 &&
                  (reinterpret_cast<uintptr_t>(bank_maps) & 127u) == 0 && (reinterpret_cast<uintptr_t>(shared_maps) & 127u) == 0,
              kMisaligned, "moe_grouped: misaligned buffer (scratch 256 bytes, descriptors 128, x and outputs 16)");
  if (tokens == 0) return kOk;
  cudaStream_t s = (cudaStream_t)stream;
  const GgScratch in(fp4, routes, groups, hidden), act(fp4, routes, groups, intermediate);
  unsigned char* p = (unsigned char*)scratch;
  auto take = [&](size_t n) { unsigned char* q = p; p += gg_pad256(n); return q; };
  unsigned char *in_image = take(in.image), *in_scales = take(in.image_scales), *in_slot = take(in.slot_scale), *in_next = take(in.next);
  unsigned char *act_image = take(act.image), *act_scales = take(act.image_scales), *act_slot = take(act.slot_scale), *act_next = take(act.next);
  unsigned char *x_image = take(n_shared ? padded * hidden * 2 : 0), *sact_image = take(padded * n_shared * intermediate * 2);
  unsigned char* shared_out = take((size_t)tokens * n_shared * hidden * 2);
  const int bank = fp4 ? 3 : 1, stride = fp4 ? kBank : 2;

  StageArgs st = {};
  st.x = (const uint16_t*)x;
  st.pointers = pointers;
  st.experts = experts;
  st.counts = counts;
  st.rows = rows;
  st.image = in_image;
  st.image_scales = in_scales;
  st.slot_scale = (float*)in_slot;
  st.next = (unsigned*)in_next;
  st.shared_image = n_shared ? x_image : nullptr;
  st.groups = groups;
  st.capacity = capacity;
  st.stride = stride;
  st.bank = 0;
  st.k = hidden;
  st.div = top_k;
  st.tokens = tokens;
  st.tile = gg_tile(fp4, t);
  st.shared_tile = gg_tile(false, t);
  if (int rc = launch_stage(fp4, st, routes + (n_shared ? tokens : 0), s)) return rc;

  GgArgs g = {};
  g.maps = (const unsigned char*)bank_maps;
  g.pointers = pointers;
  g.experts = experts;
  g.counts = counts;
  g.rows = rows;
  g.image = in_image;
  g.image_scales = in_scales;
  g.slot_scale = (const float*)in_slot;
  g.next = (unsigned*)in_next;
  g.y = (uint16_t*)activated;
  g.groups = groups;
  g.start = start;
  g.capacity = capacity;
  g.stride = stride;
  g.bank = 0;
  g.k = hidden;
  g.n = 2 * intermediate;
  g.shared_maps = (const unsigned char*)shared_maps;
  g.shared_image = x_image;
  g.shared_y = (uint16_t*)sact_image;
  g.gammas = (const uint16_t*)gammas;
  g.n_shared = n_shared;
  g.tokens = tokens;
  g.status = status;
  if (int rc = fp4 ? launch_grouped<true, 0>(t, g, s) : launch_grouped<false, 0>(t, g, s)) return rc;

  st.x = (const uint16_t*)activated;
  st.image = act_image;
  st.image_scales = act_scales;
  st.slot_scale = (float*)act_slot;
  st.next = (unsigned*)act_next;
  st.shared_image = nullptr;
  st.bank = bank;
  st.k = intermediate;
  st.div = 1;
  st.plan_ready = 1;
  if (int rc = launch_stage(fp4, st, routes, s)) return rc;

  g.maps += fp4 ? 256 : 128;
  g.image = act_image;
  g.image_scales = act_scales;
  g.slot_scale = (const float*)act_slot;
  g.next = (unsigned*)act_next;
  g.y = (uint16_t*)down;
  g.bank = bank;
  g.k = intermediate;
  g.n = hidden;
  g.shared_maps = n_shared ? g.shared_maps + 256 : nullptr;
  g.shared_image = sact_image;
  g.shared_y = (uint16_t*)shared_out;
  if (int rc = fp4 ? launch_grouped<true, 1>(t, g, s) : launch_grouped<false, 1>(t, g, s)) return rc;

  cudaLaunchConfig_t config = {};
  config.gridDim = dim3((unsigned)tokens, (unsigned)((hidden / 8 + 255) / 256));
  config.blockDim = dim3(256);
  config.stream = s;
  cudaLaunchAttribute attribute;
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  config.attrs = &attribute;
  config.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&config, combine_kernel, (const uint16_t*)down, indices, (const uint16_t*)weights, pointers, stride, max_expert,
                                           (const uint16_t*)shared_out, n_shared, output, (uint16_t*)output_bf16, hidden, top_k, status);
  INK_REQUIRE(e == cudaSuccess, kLaunchFailed, "moe_grouped: launch failed: %s", cudaGetErrorString(e));
  return kOk;
}

// The two projections on their own, as the reference's expert_gemm calls them.
static size_t expert_gemm_tc_bytes(size_t routes, size_t groups, int k) { return GgScratch(true, routes, groups, k).total; }
extern "C" size_t ink_expert_gemm_tc_scratch_bytes(int input_rows, int k) {
  const size_t routes = 8 * (size_t)(input_rows > 0 ? input_rows : 0);   // of up to eight choices a row
  return expert_gemm_tc_bytes(routes, kGgMaxGroups, k);
}

extern "C" int ink_expert_gemm_tc(const void* x, int input_rows, const void* bank_maps, const int64_t* pointers,
                                  const int32_t* experts, const int32_t* rows, const int32_t* counts, void* y, int capacity,
                                  int n, int k, int top_k, int projection, int groups, int start, void* scratch,
                                  size_t scratch_bytes, int32_t* status, ink_stream_t stream) {
  INK_REQUIRE(x && bank_maps && pointers && experts && rows && counts && y && scratch, kBadArgument,
              "expert_gemm_tc: null pointer argument");
  INK_REQUIRE(projection == 0 || projection == 1, kBadArgument, "expert_gemm_tc: projection=%d", projection);
  if (int rc = check_grouped_shape(true, n, k, groups)) return rc;
  INK_REQUIRE(capacity >= 1 && top_k >= 1 && input_rows >= 0 && start >= 0, kBadArgument, "expert_gemm_tc: bad sizes (capacity=%d top_k=%d rows=%d)",
              capacity, top_k, input_rows);
  const size_t routes = (size_t)input_rows * (projection == 0 ? top_k : 1);   // (`capacity` bounds one group's, not all of them)
  const int t = gg_tokens((long long)routes, groups);
  if (int rc = check_items_fit(true, routes, groups, n, t)) return rc;
  INK_REQUIRE(scratch_bytes >= expert_gemm_tc_bytes(routes, groups, k), kBadArgument,
              "expert_gemm_tc: scratch of %zu bytes, %zu needed", scratch_bytes, expert_gemm_tc_bytes(routes, groups, k));
  INK_REQUIRE(aligned16(x) && aligned16(y) && aligned16(scratch) && (reinterpret_cast<uintptr_t>(bank_maps) & 127u) == 0,
              kMisaligned, "expert_gemm_tc: misaligned buffer (the descriptors need 128-byte alignment)");
  if (groups == 0 || routes == 0) return kOk;
  cudaStream_t s = (cudaStream_t)stream;
  const GgScratch sizes(true, routes, groups, k);
  StageArgs st = {};
  st.x = (const uint16_t*)x;
  st.pointers = pointers;
  st.experts = experts;
  st.counts = counts;
  st.rows = rows;
  st.image = (unsigned char*)scratch;
  st.image_scales = st.image + sizes.image;
  st.slot_scale = (float*)(st.image_scales + sizes.image_scales);
  st.next = (unsigned*)(st.image_scales + sizes.image_scales + sizes.slot_scale);
  st.groups = groups;
  st.capacity = capacity;
  st.stride = kBank;
  st.bank = projection ? 3 : 0;
  st.k = k;
  st.div = projection ? 1 : top_k;
  st.tile = gg_tile(true, t);
  st.shared_tile = gg_tile(false, t);
  if (int rc = launch_stage(true, st, routes, s)) return rc;
  GgArgs g = {};
  g.maps = (const unsigned char*)bank_maps + (projection ? 256 : 0);
  g.pointers = pointers;
  g.experts = experts;
  g.counts = counts;
  g.rows = rows;
  g.image = st.image;
  g.image_scales = st.image_scales;
  g.slot_scale = st.slot_scale;
  g.next = st.next;
  g.y = (uint16_t*)y;
  g.groups = groups;
  g.start = start;
  g.capacity = capacity;
  g.stride = kBank;
  g.bank = st.bank;
  g.k = k;
  g.n = n;
  g.status = status;
  return projection == 0 ? launch_grouped<true, 0>(t, g, s) : launch_grouped<true, 1>(t, g, s);
}
