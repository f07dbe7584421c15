// Router (sigmoid scores, top-k, BF16 weight chain) and expert plan for the resident
// placement. One launch at decode: every block computes a few logits; the block that
// finishes last turns them into indices, weights and the plan tables.
#include <stdarg.h>
#include <stdio.h>

#include "../../include/inkling_b200.h"
#include "common.cuh"

namespace ink {

static thread_local char g_error[512] = "";
void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_error, sizeof(g_error), fmt, ap);
  va_end(ap);
}

constexpr int kTokenGroup = 8;           // tokens whose accumulators a warp holds at once
constexpr int kMaxScoresPerLane = 16;    // n_routed <= 512
constexpr int kFinishThreads = 256;
constexpr int kFewTokens = 8;            // tokens the one-launch router takes
constexpr int kFusedRoutes = 32 * kFewTokens;   // their routes
constexpr int kFusedRuns = kFinishThreads / 32;
constexpr size_t kPlanSmem = 200 * 1024; // most shared memory of the plan's tables

struct RouterArgs {
  const uint16_t* x;
  const uint16_t* weight;
  const float* bias;
  const uint16_t* global_scale;
  float route_scale;
  int tokens, hidden, n_routed, n_shared, top_k;
  uint16_t* routed_logits;
  uint16_t* topk_weights;
  int64_t* topk_indices;
  uint16_t* shared_gammas;
  float* logits;           // workspace: [tokens, n_routed + n_shared] BF16-rounded logits as FP32
  float* scores;           // workspace: [tokens, n_routed] selection scores
  unsigned int* counter;   // workspace: blocks done
};

struct PlanArgs {
  const int64_t* indices;
  const int64_t* sources;
  int64_t* pointers;
  int32_t* experts;
  int32_t* counts;
  int32_t* rows;
  int start, local, stride, routes, capacity;
};

// ------------------------------------------------------------------ one token
// Executed by one warp, scores and selection in registers: lane l holds the experts l, l + 32, ... (up to 32 * K).
// A round of the selection is the lane's own best, then two hardware reductions over the warp (largest score as an
// order-preserving integer, then the lowest expert id among the lanes that hold it).
template <int K>
__device__ __forceinline__ void router_finish_token(const RouterArgs& a, int token, int* ids_out) {
  const int lane = threadIdx.x & 31;
  const int total = a.n_routed + a.n_shared;
  const float* logit = a.logits + (size_t)token * total;
  const float* scores = a.scores + (size_t)token * a.n_routed;
  float sc[K];
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const int e = i * 32 + lane;
    sc[i] = e < a.n_routed ? __ldcg(scores + e) : -INFINITY;
    if (a.routed_logits && e < a.n_routed) a.routed_logits[(size_t)token * a.n_routed + e] = (uint16_t)f32_to_bf16_bits(__ldcg(logit + e));
  }
  // top-k by repeated arg-max; ties go to the lower expert id
  int my_choice = 0;  // lane r < top_k ends up holding the r-th choice
#pragma unroll 1
  for (int r = 0; r < a.top_k; ++r) {
    float best = -INFINITY;
    int best_e = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < K; ++i) {
      if (sc[i] > best) {  // ascending e within a lane: a later equal value never replaces
        best = sc[i];
        best_e = i * 32 + lane;
      }
    }
    const unsigned bits = __float_as_uint(best + 0.f);   // (-0 counts as 0)
    const unsigned key = (bits & 0x80000000u) ? ~bits : (bits | 0x80000000u);   // a > b  <=>  key(a) > key(b)
    const unsigned top = __reduce_max_sync(0xffffffffu, key);
    int winner = (int)__reduce_min_sync(0xffffffffu, key == top ? (unsigned)best_e : 0x7fffffffu);
    if (winner == 0x7fffffff) winner = r;  // every score is -inf/NaN: fall back to a valid id
#pragma unroll
    for (int i = 0; i < K; ++i)
      if (i * 32 + lane == winner) sc[i] = -INFINITY;
    if (lane == r) my_choice = winner;
  }
  // weights over the top_k selected logits followed by the shared logits
  const int n = a.top_k + a.n_shared;
  const bool live = lane < n;
  float l = 0.f;
  if (lane < a.top_k) l = __ldcg(logit + my_choice);
  else if (live) l = __ldcg(logit + a.n_routed + (lane - a.top_k));
  // logsigmoid = min(0, x) - log1p(exp(-|x|)), result rounded to BF16
  const float lp = live ? round_bf16(fminf(0.f, l) - log1pf(__expf(-fabsf(l)))) : -INFINITY;
  float m = lp;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (fabsf(m) == INFINITY) m = 0.f;
  // logsumexp as torch composes it: exp(bf16(lp - max)) rounded, FP32 sum rounded, log rounded, + max rounded
  const float ex = live ? round_bf16(__expf(round_bf16(lp - m))) : 0.f;
  float s = ex;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  const float lse = round_bf16(round_bf16(__logf(round_bf16(s))) + m);
  float w = round_bf16(__expf(round_bf16(lp - lse)));
  w = round_bf16(w * a.route_scale);
  w = round_bf16(w * bf16_to_f32(a.global_scale[0]));
  if (lane < a.top_k) {
    a.topk_indices[(size_t)token * a.top_k + lane] = my_choice;
    a.topk_weights[(size_t)token * a.top_k + lane] = (uint16_t)f32_to_bf16_bits(w);
    if (ids_out) ids_out[token * a.top_k + lane] = my_choice;
  } else if (live) {
    a.shared_gammas[(size_t)token * a.n_shared + (lane - a.top_k)] = (uint16_t)f32_to_bf16_bits(w);
  }
}

__device__ __forceinline__ void router_finish_token(const RouterArgs& a, int token, int* ids_out) {
  if (a.n_routed <= 256) router_finish_token<8>(a, token, ids_out);
  else router_finish_token<kMaxScoresPerLane>(a, token, ids_out);
}

// ------------------------------------------------------------------------ the plan
// One block: a stable counting sort of the routes by expert. Warp w takes the w-th run of routes, counts them per expert
// (lanes with equal ids find each other with a match, so nothing is atomic), the counts become offsets by a prefix sum over
// the warps, and a second pass over the same runs hands out the places in order. `hist` is [runs][local] and `group_of`
// [local] in shared memory. (One warp per expert walking all routes took 105 us for 12 000 of them, the compare loop of a
// single block 18 us for 366; this one is two passes over routes / 1024 steps.)
constexpr int kPlanRuns = 32;
__device__ void plan_block(const PlanArgs& p, const int* ids, int* hist, int* group_of, int* warp_totals, int runs) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
  const int per_run = ((p.routes + runs - 1) / runs + 31) / 32 * 32;
  auto id_of = [&](int r, int end) -> int {   // local id, -1: not on this rank
    if (r >= end) return -1;
    const int64_t id = ids ? (int64_t)ids[r] : __ldcg(p.indices + r);
    return (id >= p.start && id < (int64_t)p.start + p.local) ? (int)(id - p.start) : -1;
  };
  for (int i = tid; i < runs * p.local; i += blockDim.x) hist[i] = 0;
  __syncthreads();
  const int first = warp * per_run, end = min(p.routes, first + per_run);
  if (warp < runs) {
    int* mine = hist + warp * p.local;
    int next = id_of(first + lane, end);
    for (int r = first; r < end; r += 32) {
      const int id = next;
      next = id_of(r + 32 + lane, end);
      const unsigned same = __match_any_sync(0xffffffffu, id);
      if (id >= 0 && lane == __ffs(same) - 1) mine[id] += __popc(same);
      __syncwarp();
    }
  }
  __syncthreads();
  int groups_before = 0;
  for (int base = 0; base < p.local; base += blockDim.x) {
    const int e = base + tid;
    int count = 0;
    if (e < p.local) {
      for (int w = 0; w < runs; ++w) {
        const int n = hist[w * p.local + e];
        hist[w * p.local + e] = count;
        count += n;
      }
    }
    const bool active = count > 0;
    const unsigned ballot = __ballot_sync(0xffffffffu, active);
    if (lane == 0) warp_totals[warp] = __popc(ballot);
    __syncthreads();
    int before = groups_before, chunk_total = 0;
    for (int w = 0; w < warps; ++w) {
      if (w < warp) before += warp_totals[w];
      chunk_total += warp_totals[w];
    }
    const int group = before + __popc(ballot & ((1u << lane) - 1u));
    if (e < p.local) {
      group_of[e] = group;
      if (active) {
        p.experts[group] = p.start + e;
        p.counts[group] = count;
      }
      for (int b = 0; b < p.stride; ++b)
        p.pointers[(size_t)(p.start + e) * p.stride + b] = active ? p.sources[(size_t)e * p.stride + b] : 0;
    }
    groups_before += chunk_total;
    __syncthreads();
  }
  for (int g = groups_before + tid; g < p.local; g += blockDim.x) {
    p.experts[g] = -1;
    p.counts[g] = 0;
  }
  if (warp < runs) {
    int* mine = hist + warp * p.local;
    int next = id_of(first + lane, end);
    for (int r = first; r < end; r += 32) {
      const int id = next;
      next = id_of(r + 32 + lane, end);
      const unsigned same = __match_any_sync(0xffffffffu, id);
      int at = 0;
      if (id >= 0) at = mine[id] + __popc(same & ((1u << lane) - 1u));
      __syncwarp();
      if (id >= 0) {
        p.rows[(size_t)group_of[id] * p.capacity + at] = r + lane;
        if (lane == __ffs(same) - 1) mine[id] += __popc(same);
      }
      __syncwarp();
    }
  }
}

// ------------------------------------------------------------------- logits kernel
// kRowsPerBlock rows of the router weight per block, kWarpsPerRow warps per row, so a
// 4096-wide row is one round trip of four 16-byte loads per thread. TG tokens share
// one pass over the row.
constexpr int kRowsPerBlock = 2;
constexpr int kWarpsPerRow = kFinishThreads / 32 / kRowsPerBlock;

template <bool kFusePlan, int TG>
__global__ void __launch_bounds__(kFinishThreads) router_kernel(RouterArgs a, PlanArgs p) {
  __shared__ int s_ids[kFusedRoutes];
  __shared__ int s_warp_totals[32];
  __shared__ int s_hist[kFusePlan ? kFusedRuns * 32 * kMaxScoresPerLane : 1], s_group_of[kFusePlan ? 32 * kMaxScoresPerLane : 1];
  __shared__ float s_part[kRowsPerBlock][kWarpsPerRow][TG];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int total = a.n_routed + a.n_shared;
  const int local_row = warp / kWarpsPerRow, part = warp % kWarpsPerRow;
  const int row = blockIdx.x * kRowsPerBlock + local_row;
  const int chunks = a.hidden / 8;  // 16-byte chunks per row
  for (int t0 = 0; t0 < a.tokens; t0 += TG) {
    float acc[TG];
#pragma unroll
    for (int t = 0; t < TG; ++t) acc[t] = 0.f;
    if (row < total) {
      const uint4* w = reinterpret_cast<const uint4*>(a.weight + (size_t)row * a.hidden);
#pragma unroll 4
      for (int c = part * 32 + lane; c < chunks; c += 32 * kWarpsPerRow) {
        const uint4 q = __ldg(w + c);
#pragma unroll
        for (int t = 0; t < TG; ++t) {
          if (t0 + t < a.tokens) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(a.x + (size_t)(t0 + t) * a.hidden) + c);
            float s = acc[t];
            s = fmaf(bf16lo(q.x), bf16lo(v.x), s);
            s = fmaf(bf16hi(q.x), bf16hi(v.x), s);
            s = fmaf(bf16lo(q.y), bf16lo(v.y), s);
            s = fmaf(bf16hi(q.y), bf16hi(v.y), s);
            s = fmaf(bf16lo(q.z), bf16lo(v.z), s);
            s = fmaf(bf16hi(q.z), bf16hi(v.z), s);
            s = fmaf(bf16lo(q.w), bf16lo(v.w), s);
            s = fmaf(bf16hi(q.w), bf16hi(v.w), s);
            acc[t] = s;
          }
        }
      }
    }
#pragma unroll
    for (int t = 0; t < TG; ++t) {
      const float s = warp_sum(acc[t]);
      if (lane == 0) s_part[local_row][part][t] = s;
    }
    __syncthreads();
    if (threadIdx.x < kRowsPerBlock * TG) {
      const int r = threadIdx.x / TG, t = threadIdx.x % TG;
      const int out_row = blockIdx.x * kRowsPerBlock + r;
      if (out_row < total && t0 + t < a.tokens) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < kWarpsPerRow; ++w) s += s_part[r][w][t];
        const float l = round_bf16(s);
        a.logits[(size_t)(t0 + t) * total + out_row] = l;
        // BF16 sigmoid, then FP32 add of the FP32 bias: the value the top-k compares
        if (out_row < a.n_routed)
          a.scores[(size_t)(t0 + t) * a.n_routed + out_row] = round_bf16(1.f / (1.f + __expf(-l))) + a.bias[out_row];
      }
    }
    __syncthreads();
  }
  // the block that arrives last owns the tail of the computation
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned done = atomicAdd(a.counter, 1u);
    s_last = (done == gridDim.x - 1);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int token = warp; token < a.tokens; token += warps)
    router_finish_token(a, token, kFusePlan ? s_ids : nullptr);
  if (kFusePlan) {
    __syncthreads();
    plan_block(p, s_ids, s_hist, s_group_of, s_warp_totals, kFusedRuns);
  }
  if (threadIdx.x == 0) *a.counter = 0u;  // leave the workspace ready for the next call
}

__global__ void __launch_bounds__(1024) plan_kernel(PlanArgs p, int runs) {
  extern __shared__ int s_plan[];   // [runs][local] counts, [local] groups
  __shared__ int s_warp_totals[32];
  plan_block(p, nullptr, s_plan, s_plan + runs * p.local, s_warp_totals, runs);
}

// ------------------------------------------------------------- router, many tokens
// The logits of more than a handful of tokens: a block takes tiles of sixteen router rows and sixteen tokens, a thread the partial
// sums of sixteen tokens and half of the rows over its columns. A thread's columns, the order of its sums and the order in which the
// threads' sums are added are those of router_kernel, so a token's logits do not depend on how many others there are (the
// selection compares BF16 values: a last-bit difference picks another expert): products on the CUDA cores, two rows' FMAs an instruction.
// Persistent blocks, one an SM: the next chunks of columns, of this tile or the next, are copied to shared memory while one is computed on.
// 1 999 tokens, 258 rows of 4 096 columns (2.1 G FMAs, 58 us at the FMA pipes' rate): 160 us, 52 % of the issue slots, 2.6 instructions
// for each that multiplies (tokens spread to pairs, the sums over the threads); router_kernel, two rows a block and its tail on one block, 3 270.
// Loads straight to registers (router_logits_tile_kernel, which was here for all tiles) depend on where the operands are. In DRAM, as a block's
// experts leave them: a block of 4096 x 512 with 256 experts 707 us at 1 999 tokens and 426 at 926, 672 and 406 so. The tokens in L2, written just
// before: 659 and 403, 680 and 409 so. Tokens and weights in L2, the router alone called again and again: 135 at 1 999 tokens, 166 so.
constexpr int kManyRows = 8, kManyTokens = 16, kManyGroups = 2;            // rows of a thread, tokens, threads' shares of a tile's rows
constexpr int kManyColumns = 128;                                           // threads along the columns, eight of them each
constexpr int kManyThreads = kManyGroups * kManyColumns;
constexpr int kManyTileRows = kManyGroups * kManyRows;
constexpr int kManyStages = 3;
constexpr int kManyStageBytes = (kManyTileRows + kManyTokens) * kManyColumns * 16;
constexpr int kManySmem = kManyStages * kManyStageBytes;

// Sums N per-lane values over the warp in the order of warp_sum; lane l keeps the values first, first + 1, ... (N / 32).
template <int N>
__device__ __forceinline__ int wide_reduce(float (&v)[N], int lane) {
  int first = 0;
#pragma unroll
  for (int o = 16, n = N; o > 0; o >>= 1, n >>= 1) {
    const bool upper = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < n / 2; ++i) {
      const float send = upper ? v[i] : v[i + n / 2];
      const float keep = upper ? v[i + n / 2] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
    first += upper ? n / 2 : 0;
  }
  return first;
}

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// The logit of pair `i` of a tile, of this row and token, from the warps' sums of it.
template <int PARTS>
__device__ __forceinline__ void write_logit(const RouterArgs& a, const float (&part)[PARTS][kManyRows * kManyTokens], int i, int row, int token) {
  static_assert(kManyRows * kManyTokens == kManyColumns, "a thread writes one logit");
  if (row >= a.n_routed + a.n_shared || token >= a.tokens) return;
  float s = 0.f;
#pragma unroll
  for (int w = 0; w < PARTS; ++w) s += part[w][i];
  const float l = round_bf16(s);
  a.logits[(size_t)token * (a.n_routed + a.n_shared) + row] = l;
  if (row < a.n_routed) a.scores[(size_t)token * a.n_routed + row] = round_bf16(1.f / (1.f + __expf(-l))) + a.bias[row];
}

// One tile of tokens (nine to sixteen): no next tile to copy ahead, and half as many rows a block put twice as many SMs to work. Loads go
// straight to registers; rows and tokens are asked for into L2 all at once, where the router's weights rarely are.
__global__ void __launch_bounds__(kManyColumns, 2) router_logits_tile_kernel(RouterArgs a) {
  constexpr int kPairs = kManyRows * kManyTokens, kParts = kManyColumns / 32;
  __shared__ float s_part[kParts][kPairs];
  const int tid = threadIdx.x, lane = tid & 31, part = tid >> 5;
  const int total = a.n_routed + a.n_shared, chunks = a.hidden / 8, row0 = blockIdx.x * kManyRows;
  const size_t row_bytes = (size_t)a.hidden * 2, w_bytes = min(kManyRows, total - row0) * row_bytes, x_bytes = a.tokens * row_bytes;
  const char *w_from = reinterpret_cast<const char*>(a.weight) + row0 * row_bytes, *x_from = reinterpret_cast<const char*>(a.x);
  for (size_t i = (size_t)tid * 128; i < w_bytes; i += kManyColumns * 128) prefetch_l2(w_from + i);
  for (size_t i = ((size_t)blockIdx.x * kManyColumns + tid) * 128; i < x_bytes; i += (size_t)gridDim.x * kManyColumns * 128) prefetch_l2(x_from + i);
  float acc[kPairs];   // [token][row]
#pragma unroll
  for (int i = 0; i < kPairs; ++i) acc[i] = 0.f;
#pragma unroll 1
  for (int c = tid; c < chunks; c += kManyColumns) {
    float w[kManyRows][8];
#pragma unroll
    for (int r = 0; r < kManyRows; ++r) {
      const uint4 q = __ldg(reinterpret_cast<const uint4*>(a.weight + (size_t)min(row0 + r, total - 1) * a.hidden) + c);
      w[r][0] = bf16lo(q.x); w[r][1] = bf16hi(q.x); w[r][2] = bf16lo(q.y); w[r][3] = bf16hi(q.y);
      w[r][4] = bf16lo(q.z); w[r][5] = bf16hi(q.z); w[r][6] = bf16lo(q.w); w[r][7] = bf16hi(q.w);
    }
#pragma unroll
    for (int t0 = 0; t0 < kManyTokens; t0 += 4) {
      uint4 x4[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) x4[t] = __ldg(reinterpret_cast<const uint4*>(a.x + (size_t)min(t0 + t, a.tokens - 1) * a.hidden) + c);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float x[8] = {bf16lo(x4[t].x), bf16hi(x4[t].x), bf16lo(x4[t].y), bf16hi(x4[t].y),
                            bf16lo(x4[t].z), bf16hi(x4[t].z), bf16lo(x4[t].w), bf16hi(x4[t].w)};
#pragma unroll
        for (int r = 0; r < kManyRows; ++r)
#pragma unroll
          for (int k = 0; k < 8; ++k) acc[(t0 + t) * kManyRows + r] = fmaf(w[r][k], x[k], acc[(t0 + t) * kManyRows + r]);
      }
    }
  }
  const int first = wide_reduce<kPairs>(acc, lane);
#pragma unroll
  for (int i = 0; i < kPairs / 32; ++i) s_part[part][first + i] = acc[i];
  __syncthreads();
  write_logit<kParts>(a, s_part, tid, row0 + tid % kManyRows, tid / kManyRows);
}

__device__ __forceinline__ uint64_t pair_of(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__global__ void __launch_bounds__(kManyThreads, 1) router_logits_kernel(RouterArgs a) {
  constexpr int kPairs = kManyRows * kManyTokens, kParts = kManyColumns / 32, kRowPairs = kManyRows / 2;
  extern __shared__ __align__(16) unsigned char s_many[];   // [stages][sixteen rows, sixteen tokens][columns][16 B]
  __shared__ float s_part[kManyGroups][kParts][kPairs];
  const int tid = threadIdx.x, lane = tid & 31, group = tid / kManyColumns, column = tid % kManyColumns, part = column >> 5;
  const int total = a.n_routed + a.n_shared, pieces = a.hidden / 8, chunks = (pieces + kManyColumns - 1) / kManyColumns;
  const int row_tiles = (total + kManyTileRows - 1) / kManyTileRows;
  const long long tiles = (long long)row_tiles * (a.tokens / kManyTokens + (a.tokens % kManyTokens != 0));
  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(s_many);
  // the copies of one chunk of a tile, half of its rows each: a group of copies (maybe an empty one)
  long long copy_tile = blockIdx.x;
  int copy_chunk = 0, copy_stage = 0;
  auto copy_next = [&]() {
    if (copy_tile < tiles) {
      const int row0 = (int)(copy_tile % row_tiles) * kManyTileRows, token0 = (int)(copy_tile / row_tiles) * kManyTokens;
      const int piece = copy_chunk * kManyColumns + column;
      const uint32_t to = ring + (uint32_t)(copy_stage * kManyStageBytes + column * 16);
#pragma unroll 4
      for (int r = group; r < kManyTileRows + kManyTokens; r += kManyGroups) {
        const uint16_t* from = r < kManyTileRows ? a.weight + (size_t)min(row0 + r, total - 1) * a.hidden
                                                 : a.x + (size_t)min(token0 + r - kManyTileRows, a.tokens - 1) * a.hidden;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + (uint32_t)(r * kManyColumns * 16)),
                     "l"(from + (piece < pieces ? piece * 8 : 0)), "r"(piece < pieces ? 16 : 0)   // (0: zeros, which add nothing)
                     : "memory");
      }
      copy_stage = (copy_stage + 1) % kManyStages;
      if (++copy_chunk == chunks) {
        copy_chunk = 0;
        copy_tile += gridDim.x;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int i = 0; i + 1 < kManyStages; ++i) copy_next();
  int stage = 0;
  for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int row0 = (int)(tile % row_tiles) * kManyTileRows + group * kManyRows, token0 = (int)(tile / row_tiles) * kManyTokens;
    uint64_t acc2[kManyTokens][kRowPairs];   // sums of two rows
#pragma unroll
    for (int t = 0; t < kManyTokens; ++t)
#pragma unroll
      for (int r = 0; r < kRowPairs; ++r) acc2[t][r] = 0ull;
#pragma unroll 1
    for (int c = 0; c < chunks; ++c) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kManyStages - 2) : "memory");
      __syncthreads();   // everybody's copies of this chunk are there, everybody is done with the one before
      copy_next();
      const unsigned char* at = s_many + stage * kManyStageBytes + column * 16;
      stage = (stage + 1) % kManyStages;
      uint64_t w[kRowPairs][8];
#pragma unroll
      for (int r = 0; r < kRowPairs; ++r) {
        const uint4 q0 = *reinterpret_cast<const uint4*>(at + (group * kManyRows + 2 * r) * kManyColumns * 16);
        const uint4 q1 = *reinterpret_cast<const uint4*>(at + (group * kManyRows + 2 * r + 1) * kManyColumns * 16);
        const uint32_t v0[4] = {q0.x, q0.y, q0.z, q0.w}, v1[4] = {q1.x, q1.y, q1.z, q1.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          w[r][2 * k] = pair_of(bf16lo(v0[k]), bf16lo(v1[k]));
          w[r][2 * k + 1] = pair_of(bf16hi(v0[k]), bf16hi(v1[k]));
        }
      }
      constexpr int kAtOnce = 4;   // tokens: sixteen sums that do not wait for one another
#pragma unroll
      for (int t0 = 0; t0 < kManyTokens; t0 += kAtOnce) {
        uint32_t v[kAtOnce][4];
#pragma unroll
        for (int t = 0; t < kAtOnce; ++t) {
          const uint4 q = *reinterpret_cast<const uint4*>(at + (kManyTileRows + t0 + t) * kManyColumns * 16);
          v[t][0] = q.x; v[t][1] = q.y; v[t][2] = q.z; v[t][3] = q.w;
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
#pragma unroll
          for (int t = 0; t < kAtOnce; ++t) {
            const float x = (k & 1) ? bf16hi(v[t][k / 2]) : bf16lo(v[t][k / 2]);
            const uint64_t xx = pair_of(x, x);
#pragma unroll
            for (int r = 0; r < kRowPairs; ++r) asm volatile("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc2[t0 + t][r]) : "l"(w[r][k]), "l"(xx));
          }
        }
      }
    }
    float acc[kPairs];   // [token][row]
#pragma unroll
    for (int t = 0; t < kManyTokens; ++t)
#pragma unroll
      for (int r = 0; r < kRowPairs; ++r) asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[t * kManyRows + 2 * r]), "=f"(acc[t * kManyRows + 2 * r + 1]) : "l"(acc2[t][r]));
    const int first = wide_reduce<kPairs>(acc, lane);
#pragma unroll
    for (int i = 0; i < kPairs / 32; ++i) s_part[group][part][first + i] = acc[i];
    __syncthreads();   // (the next tile's first barrier keeps these sums until they have been read)
    write_logit<kParts>(a, s_part[group], column, row0 + column % kManyRows, token0 + column / kManyRows);   // a pair a thread
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// One warp per token; the block that is done last makes the plan, if one is asked for.
template <bool kFusePlan>
__global__ void __launch_bounds__(1024) router_select_kernel(RouterArgs a, PlanArgs p, int runs) {
  extern __shared__ int s_plan[];
  __shared__ int s_warp_totals[32];
  __shared__ bool s_last;
  const int token = blockIdx.x * 32 + (threadIdx.x >> 5);
  if (token < a.tokens) router_finish_token(a, token, nullptr);
  if (!kFusePlan) return;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    s_last = atomicAdd(a.counter, 1u) == gridDim.x - 1;
    if (s_last) *a.counter = 0u;   // leave the workspace ready for the next call
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  plan_block(p, nullptr, s_plan, s_plan + runs * p.local, s_warp_totals, runs);
}

static int check_router(const RouterArgs& a, size_t workspace_bytes) {
  INK_REQUIRE(a.tokens >= 0 && a.hidden > 0, kBadArgument, "router: tokens=%d hidden=%d", a.tokens, a.hidden);
  INK_REQUIRE(a.hidden % 8 == 0, kUnsupportedShape, "router: hidden=%d must be a multiple of 8", a.hidden);
  INK_REQUIRE(a.n_routed > 0 && a.n_routed <= 32 * kMaxScoresPerLane, kUnsupportedShape,
              "router: n_routed=%d must be between 1 and %d", a.n_routed, 32 * kMaxScoresPerLane);
  INK_REQUIRE(a.top_k >= 1 && a.top_k <= 32 && a.top_k <= a.n_routed && a.n_shared >= 0 && a.top_k + a.n_shared <= 32,
              kUnsupportedShape, "router: top_k=%d n_shared=%d unsupported", a.top_k, a.n_shared);
  INK_REQUIRE(a.x && a.weight && a.bias && a.global_scale && a.topk_weights && a.topk_indices &&
                  (a.n_shared == 0 || a.shared_gammas) && a.logits,
              kBadArgument, "router: null pointer argument");
  INK_REQUIRE(aligned16(a.x) && aligned16(a.weight), kMisaligned, "router: x and weight must be 16-byte aligned");
  INK_REQUIRE(workspace_bytes >= ink_router_workspace_bytes(a.tokens, a.n_routed + a.n_shared), kBadArgument,
              "router: workspace of %zu bytes is too small", workspace_bytes);
  return kOk;
}

static int check_plan(const PlanArgs& p) {
  INK_REQUIRE(p.indices && p.sources && p.pointers && p.experts && p.counts && p.rows, kBadArgument,
              "expert_plan: null pointer argument");
  INK_REQUIRE(p.local > 0 && p.start >= 0 && p.stride > 0 && p.routes >= 0 && p.capacity >= 1, kBadArgument,
              "expert_plan: start=%d local=%d stride=%d routes=%d capacity=%d", p.start, p.local, p.stride,
              p.routes, p.capacity);
  INK_REQUIRE((size_t)p.local * 2 * sizeof(int) <= kPlanSmem, kUnsupportedShape, "expert_plan: %d experts on this rank", p.local);
  return kOk;
}

// Runs of routes the plan sorts side by side: as many warps as have a step's worth, as far as their tables fit.
static int plan_runs(const PlanArgs& p) {
  const int fit = (int)(kPlanSmem / sizeof(int) / p.local) - 1, whole = (p.routes + 31) / 32;
  const int runs = fit < kPlanRuns ? fit : kPlanRuns;
  return whole < 1 ? 1 : whole < runs ? whole : runs;
}
template <typename Kernel>
static int allow_plan_smem(Kernel kernel) {
  constexpr int kMaxDevices = 64;
  static bool done[kMaxDevices] = {};
  int device = 0;
  cudaGetDevice(&device);
  INK_REQUIRE(device >= 0 && device < kMaxDevices, kLaunchFailed, "expert_plan: device ordinal %d", device);
  if (!done[device]) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPlanSmem);
    INK_REQUIRE(e == cudaSuccess, kLaunchFailed, "expert_plan: shared memory opt-in refused: %s", cudaGetErrorString(e));
    done[device] = true;
  }
  return kOk;
}

// The router, with the plan if `p` is given. Up to eight tokens: one launch, whose last block selects and plans; more: the
// logits by themselves (the last block of one launch would select for thousands of tokens alone), then selection and plan.
static int launch_router(const RouterArgs& a, const PlanArgs* p, cudaStream_t stream) {
  const int rows = a.n_routed + a.n_shared, blocks = (rows + kRowsPerBlock - 1) / kRowsPerBlock;
  if (a.tokens <= kFewTokens && (!p || p->local <= 32 * kMaxScoresPerLane)) {
    const PlanArgs plan = p ? *p : PlanArgs{};
    if (p && a.tokens == 1) router_kernel<true, 1><<<blocks, kFinishThreads, 0, stream>>>(a, plan);
    else if (p) router_kernel<true, kTokenGroup><<<blocks, kFinishThreads, 0, stream>>>(a, plan);
    else if (a.tokens == 1) router_kernel<false, 1><<<blocks, kFinishThreads, 0, stream>>>(a, plan);
    else router_kernel<false, kTokenGroup><<<blocks, kFinishThreads, 0, stream>>>(a, plan);
    INK_CHECK_LAUNCH("ink_router_forward");
    return kOk;
  }
  constexpr int kMaxDevices = 64;
  static int sms_of[kMaxDevices] = {};   // 0: this device is not configured yet
  int device = 0;
  cudaGetDevice(&device);
  INK_REQUIRE(device >= 0 && device < kMaxDevices, kLaunchFailed, "router: device ordinal %d", device);
  if (a.tokens > kManyTokens && sms_of[device] == 0) {
    const cudaError_t e = cudaFuncSetAttribute(router_logits_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kManySmem);
    INK_REQUIRE(e == cudaSuccess, kLaunchFailed, "router: %d bytes of shared memory refused: %s", kManySmem, cudaGetErrorString(e));
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    sms_of[device] = sms > 0 ? sms : 148;
  }
  // us, register loads / persistent: alone, all in L2, 9 tokens 10.3 / 14.6 and 16 tokens 11.3 / 14.9 (so with the prefetch 11.0 and 11.5); a block
  // of 4096 x 512, 256 experts, tokens in DRAM: 9 tokens 74.5 / 75.3, 16 tokens 83.8 / 84.2, 30 tokens 103.5 / 102.4, 63 tokens 135.7 / 134.4.
  if (a.tokens <= kManyTokens) {
    router_logits_tile_kernel<<<(rows + kManyRows - 1) / kManyRows, kManyColumns, 0, stream>>>(a);
  } else {
    const long long tiles = (long long)((rows + kManyTileRows - 1) / kManyTileRows) * ((a.tokens + (long long)kManyTokens - 1) / kManyTokens);
    router_logits_kernel<<<(unsigned)(tiles < sms_of[device] ? tiles : sms_of[device]), kManyThreads, kManySmem, stream>>>(a);
  }
  INK_CHECK_LAUNCH("ink_router_forward (logits)");
  const unsigned selects = (unsigned)((a.tokens + 31) / 32);
  if (!p) {
    router_select_kernel<false><<<selects, 1024, 0, stream>>>(a, PlanArgs{}, 0);
  } else {
    if (int rc = allow_plan_smem(router_select_kernel<true>)) return rc;
    const int runs = plan_runs(*p);
    router_select_kernel<true><<<selects, 1024, sizeof(int) * (size_t)(runs + 1) * p->local, stream>>>(a, *p, runs);
  }
  INK_CHECK_LAUNCH("ink_router_forward (selection)");
  return kOk;
}

}  // namespace ink

using namespace ink;

extern "C" const char* ink_last_error(void) { return g_error; }
extern "C" int ink_abi_version(void) { return 1; }

extern "C" size_t ink_router_workspace_bytes(int tokens, int n_experts_total) {
  // 256 bytes of counters, then the FP32 logits and the FP32 selection scores
  return 256 + 2 * sizeof(float) * (size_t)(tokens > 0 ? tokens : 0) * (size_t)n_experts_total;
}

static RouterArgs make_router_args(const void* x, const void* weight, const float* bias, const void* global_scale,
                                   float route_scale, int tokens, int hidden, int n_routed, int n_shared,
                                   int top_k, void* routed_logits, void* topk_weights, int64_t* topk_indices,
                                   void* shared_gammas, void* workspace) {
  RouterArgs a;
  a.x = (const uint16_t*)x;
  a.weight = (const uint16_t*)weight;
  a.bias = bias;
  a.global_scale = (const uint16_t*)global_scale;
  a.route_scale = route_scale;
  a.tokens = tokens;
  a.hidden = hidden;
  a.n_routed = n_routed;
  a.n_shared = n_shared;
  a.top_k = top_k;
  a.routed_logits = (uint16_t*)routed_logits;
  a.topk_weights = (uint16_t*)topk_weights;
  a.topk_indices = topk_indices;
  a.shared_gammas = (uint16_t*)shared_gammas;
  a.counter = (unsigned int*)workspace;
  a.logits = workspace ? (float*)((char*)workspace + 256) : nullptr;
  a.scores = a.logits ? a.logits + (size_t)(tokens > 0 ? tokens : 0) * (size_t)(n_routed + n_shared) : nullptr;
  return a;
}

extern "C" int ink_router_forward(const void* x, const void* weight, const float* bias, const void* global_scale,
                                  float route_scale, int tokens, int hidden, int n_routed, int n_shared,
                                  int top_k, void* routed_logits, void* topk_weights, int64_t* topk_indices,
                                  void* shared_gammas, void* workspace, size_t workspace_bytes,
                                  ink_stream_t stream) {
  RouterArgs a = make_router_args(x, weight, bias, global_scale, route_scale, tokens, hidden, n_routed, n_shared,
                                  top_k, routed_logits, topk_weights, topk_indices, shared_gammas, workspace);
  if (int rc = check_router(a, workspace_bytes)) return rc;
  if (tokens == 0) return kOk;
  return launch_router(a, nullptr, (cudaStream_t)stream);
}

// ------------------------------------------------------------ router, no allocation
// Scratch for ink_router_forward_static: lives in the library image, so a process that
// loads the library holds these bytes on every GPU it uses, until it exits.
constexpr int kStaticRouterTokens = 8;
constexpr int kStaticRouterExperts = 32 * kMaxScoresPerLane + 32;   // routed + shared rows at most
constexpr size_t kStaticRouterBytes = 256 + 2 * sizeof(float) * kStaticRouterTokens * kStaticRouterExperts;
static __device__ __align__(256) unsigned char g_static_router_scratch[kStaticRouterBytes];

constexpr int kStaticMaxDevices = 64;
// Device address of the array, per device ordinal. Written without a lock: two host threads that
// make the first call on a device together both look the address up and store the same value.
// The address stays valid for the life of the process as long as the device is not reset.
static void* g_static_router_ptr[kStaticMaxDevices];

extern "C" int ink_router_forward_static(const void* x, const void* weight, const float* bias,
                                         const void* global_scale, float route_scale, int tokens, int hidden,
                                         int n_routed, int n_shared, int top_k, void* routed_logits,
                                         void* topk_weights, int64_t* topk_indices, void* shared_gammas,
                                         ink_stream_t stream) {
  INK_REQUIRE(tokens >= 0 && tokens <= kStaticRouterTokens, kUnsupportedShape,
              "router (static scratch): %d tokens, the built-in scratch holds at most %d", tokens,
              kStaticRouterTokens);
  INK_REQUIRE(n_routed > 0 && n_shared >= 0 && n_routed + n_shared <= kStaticRouterExperts, kUnsupportedShape,
              "router (static scratch): %d router rows, the built-in scratch holds at most %d",
              n_routed + n_shared, kStaticRouterExperts);
  int device = -1;
  cudaError_t e = cudaGetDevice(&device);
  INK_REQUIRE(e == cudaSuccess && device >= 0 && device < kStaticMaxDevices, kLaunchFailed,
              "router (static scratch): cannot identify the current device: %s", cudaGetErrorString(e));
  if (g_static_router_ptr[device] == nullptr) {
    // The array's name is only a handle on the host: ask the runtime for its address on
    // the device that is current now, once, and keep it.
    void* address = nullptr;
    e = cudaGetSymbolAddress(&address, g_static_router_scratch);
    INK_REQUIRE(e == cudaSuccess && address != nullptr, kLaunchFailed,
                "router (static scratch): cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
    g_static_router_ptr[device] = address;
  }
  void* scratch = g_static_router_ptr[device];
  // The block counter at the head of the scratch must be zero when the kernel starts; the
  // previous call normally leaves it so, but a call that was cut short would not.
  e = cudaMemsetAsync(scratch, 0, 256, (cudaStream_t)stream);
  INK_REQUIRE(e == cudaSuccess, kLaunchFailed, "router (static scratch): memset failed: %s", cudaGetErrorString(e));
  return ink_router_forward(x, weight, bias, global_scale, route_scale, tokens, hidden, n_routed, n_shared, top_k,
                            routed_logits, topk_weights, topk_indices, shared_gammas, scratch, kStaticRouterBytes,
                            stream);
}

extern "C" int ink_router_plan_forward(const void* x, const void* weight, const float* bias,
                                       const void* global_scale, float route_scale, int tokens, int hidden,
                                       int n_routed, int n_shared, int top_k, void* routed_logits,
                                       void* topk_weights, int64_t* topk_indices, void* shared_gammas,
                                       void* workspace, size_t workspace_bytes, const int64_t* sources,
                                       int64_t* pointers, int32_t* experts, int32_t* counts, int32_t* rows,
                                       int start, int local, int stride, int capacity, ink_stream_t stream) {
  RouterArgs a = make_router_args(x, weight, bias, global_scale, route_scale, tokens, hidden, n_routed, n_shared,
                                  top_k, routed_logits, topk_weights, topk_indices, shared_gammas, workspace);
  if (int rc = check_router(a, workspace_bytes)) return rc;
  PlanArgs p{topk_indices, sources, pointers, experts, counts, rows, start, local, stride, tokens * top_k, capacity};
  if (int rc = check_plan(p)) return rc;
  INK_REQUIRE(capacity >= p.routes || capacity >= tokens, kBadArgument, "router_plan: capacity=%d too small", capacity);
  if (tokens == 0) return kOk;
  return launch_router(a, &p, (cudaStream_t)stream);
}

extern "C" int ink_expert_plan(const int64_t* indices, const int64_t* sources, int64_t* pointers,
                               int32_t* experts, int32_t* counts, int32_t* rows, int start, int local,
                               int stride, int routes, int capacity, ink_stream_t stream) {
  PlanArgs p{indices, sources, pointers, experts, counts, rows, start, local, stride, routes, capacity};
  if (int rc = check_plan(p)) return rc;
  if (int rc = allow_plan_smem(plan_kernel)) return rc;
  const int runs = plan_runs(p);
  plan_kernel<<<1, 1024, sizeof(int) * (size_t)(runs + 1) * local, (cudaStream_t)stream>>>(p, runs);
  INK_CHECK_LAUNCH("ink_expert_plan");
  return kOk;
}
