// Decode attention with the learned relative-position bias: one query token per sequence against the
// layer's K/V cache (a ring of `window` slots in a sliding layer, `slots` positions in a full one).
#include "../../include/inkling_b200.h"
#include "common.cuh"
#include "mma_bf16.cuh"
#include "stream_math.cuh"

namespace ink {

constexpr int kAttnThreads = 128;
constexpr int kAttnWarps = kAttnThreads / 32;
constexpr int kAttnHeads = 8;                               // query heads that share a pass over the cache rows
constexpr int kAttnUnit = 16;                               // cache slots per step of a warp
constexpr int kAttnMinSlots = kAttnUnit * kAttnWarps;       // a block is not worth launching for fewer
constexpr int kAttnCluster = 8;                             // parts that can meet in one thread-block cluster
constexpr int kAttnMaxSplits = 64;
// Blocks of the large form that an SM holds, and clusters of n = 0, 1, .. 8 parts that are resident at once on 148 SMs
// (cudaOccupancyMaxActiveClusters: a cluster lies in one GPC, so those of seven or eight parts leave a tenth of the SMs empty).
constexpr int kAttnPerSm(int channels) { return channels > 128 ? 2 : 3; }
constexpr int kAttnSms = 148;
constexpr int kAttnClusters[2][kAttnCluster + 1] = {{0, 444, 222, 142, 104, 82, 71, 56, 48}, {0, 296, 148, 93, 71, 56, 45, 37, 33}};
constexpr int kAttnPartial = 4;                             // floats in front of a partial result: running maximum, sum, padding

struct AttnArgs {
  const uint16_t* q;        // [bs, h, c] after q_norm
  const uint16_t* r;        // [bs, h, d_rel] relative states
  const uint16_t* proj;     // [d_rel, extent]
  const uint16_t* k;        // [bs, hk, slots, c], the current token already stored
  const uint16_t* v;
  const int64_t* position;  // device scalar: tokens stored before this one
  const int64_t* pad_counts;   // [bs] or null
  const uint16_t* new_k;    // [bs, hk, c] the current token's key and value, or null when the caches hold them already
  const uint16_t* new_v;
  uint16_t* k_store;        // the caches again, writable: where the current token is stored when new_k is given
  uint16_t* v_store;
  float* partial;           // [bs, h, splits, 4 + c]: maximum, sum of exponentials, unnormalised weighted values
  unsigned* arrived;        // [bs, head groups] blocks of a group that have stored their partial; zero between launches
  uint16_t* out;            // [bs, h, c]
  int heads, kv_heads, d_rel, extent, slots, window, n_floor, splits;
  float alpha, scale;
};

// the two floats cut off to BF16
__device__ __forceinline__ uint32_t high_halves(float lo, float hi) { return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632); }

// One block per (part of the cache, group of up to eight heads of one key/value head, sequence). Bound by reading
// the cache once: 512 bytes a slot against 32 k FMAs for eight heads of 128 channels, which the CUDA cores cannot
// deliver at HBM speed, so scores, bias and weighted values go through warp-level matrix instructions (M = heads: the
// contraction is far too flat for the 128-row tcgen05 tiles). Measured on B200, batch 8, 64 heads on 8 key/value
// heads, 30 000 of 32 768 slots: 2 586 us with one block per head and 64 slots, 171 us with this one (5.1 TB/s).
//
// A warp takes 16 slots a step and keeps everything in registers; nothing of the cache passes through shared memory,
// because the sums over channels may run in any order as long as both operands agree:
//   scores  A = the queries (row g = head), B = the keys: lane (g, t) loads the 16-byte pieces t, t + 4, ... of the row
//           of slot g; the four words of a piece are two k-steps' worth of B.
//   values  A = the exponentials, which the score accumulators already hold in A's layout; B = the values: lane (g, t)
//           loads the piece g (and g + 8) of the rows 2t, 2t+1, 2t+8, 2t+9, and word pairs of neighbouring rows are
//           interleaved into B. An exponential's 24 bits are three BF16 values, p = hi + mid + lo exactly: hi in the rows of
//           the heads, mid in the eight rows below, which nobody needs, lo by a second instruction, half of it in either
//           row (165 us without it; in any order of the instructions). The parts are cut off, not rounded, and never zero
//           beside a p that is not (2^-40 p instead, which p does not feel), so that each of them takes an infinite value
//           to the same infinity.
//
// The parts of a group of heads are joined in one of two ways. Up to eight of them form a thread-block cluster (CLUSTER)
// and read one another's sums through distributed shared memory; more leave their sums in global memory and the block that
// finishes last adds them up. The second way costs a fence, an atomic and two more round trips.
template <int C, bool CLUSTER>
__global__ void __launch_bounds__(kAttnThreads, kAttnPerSm(C)) decode_attention_kernel(AttnArgs a) {
  constexpr int kPieces = C / 32;       // 16-byte pieces of a key row per lane
  constexpr int kHalves = C / 64;       // pieces of a value row per lane
  extern __shared__ __align__(16) unsigned char s_raw[];
  float* s_acc = reinterpret_cast<float*>(s_raw);                                   // [warps][heads][C + 2]
  uint16_t* s_r = reinterpret_cast<uint16_t*>(s_raw);                               // [heads][d_rel rounded up to 16]: before the sums
  __shared__ bool s_last;
  __shared__ __align__(16) float s_block[CLUSTER ? kAttnHeads * (C + 2) : 1];   // this block's sums, for its cluster
  pdl_wait();
  pdl_trigger();
  const int split = blockIdx.x, b = blockIdx.z, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int group = a.heads / a.kv_heads, chunks = (group + kAttnHeads - 1) / kAttnHeads;
  const int kv_head = blockIdx.y / chunks, chunk = blockIdx.y % chunks;
  const int head0 = kv_head * group + chunk * kAttnHeads, n_heads = min(kAttnHeads, group - chunk * kAttnHeads);
  // positions fit 32 bits; the ring arithmetic is done once per block (position modulo the window), not per slot
  const int position = (int)*a.position;
  const int reach = position - (int)(a.pad_counts ? a.pad_counts[b] : 0);   // largest distance that is not padding
  const int ring_position = a.window ? position % a.window : 0;
  auto distance_of = [&](int slot) -> int {
    if (!a.window) return position - slot;
    const int d = ring_position - (slot < a.window ? slot : slot % a.window);
    return d < 0 ? d + a.window : d;
  };
  auto allowed_at = [&](int slot) -> bool {
    const int d = distance_of(slot);
    return slot < a.slots && d >= 0 && d <= reach;
  };
  const size_t row0 = ((size_t)b * a.kv_heads + kv_head) * a.slots;
  const uint16_t* keys = a.k + row0 * C;
  const uint16_t* values = a.v + row0 * C;
  // The current token may not be in the caches yet (new_k / new_v given): every block takes its row from there, and
  // one block stores it for the steps to come.
  const int fresh_slot = a.new_k ? (a.window ? ring_position : position) : -1;
  const uint16_t* fresh_k = a.new_k ? a.new_k + ((size_t)b * a.kv_heads + kv_head) * C : nullptr;
  const uint16_t* fresh_v = a.new_k ? a.new_v + ((size_t)b * a.kv_heads + kv_head) * C : nullptr;
  if (a.new_k && chunk == 0 && split == 0 && fresh_slot < a.slots) {
    for (int i = tid; i < C / 2; i += kAttnThreads) {
      reinterpret_cast<uint32_t*>(a.k_store + (row0 + fresh_slot) * C)[i] = __ldcg(reinterpret_cast<const uint32_t*>(fresh_k) + i);
      reinterpret_cast<uint32_t*>(a.v_store + (row0 + fresh_slot) * C)[i] = __ldcg(reinterpret_cast<const uint32_t*>(fresh_v) + i);
    }
  }
  // The slots that can count at all (a full layer: from the end of the padding to the position; a ring: all that have
  // been written) are dealt evenly to the splits, so that the blocks of a short context are as busy as those of a long one.
  const int lo = a.window ? 0 : max(0, position - reach);
  const int hi = (a.window == 0 || a.slots <= a.window) ? min(a.slots, position + 1) : a.slots;
  const int units = hi > lo ? (hi - lo + kAttnUnit - 1) / kAttnUnit : 0;
  const int unit0 = (int)((long long)units * split / a.splits), unit1 = (int)((long long)units * (split + 1) / a.splits);

  uint4 kq[2][kPieces];
  auto load_keys = [&](int unit) {
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int slot = lo + unit * kAttnUnit + n * 8 + g;
      const bool ok = unit < unit1 && allowed_at(slot);
      const uint4* row = reinterpret_cast<const uint4*>(slot == fresh_slot ? fresh_k : keys + (size_t)slot * C);
#pragma unroll
      for (int i = 0; i < kPieces; ++i) kq[n][i] = ok ? ld_stream_16(row + t + 4 * i) : make_uint4(0, 0, 0, 0);
    }
  };
  int unit = unit0 + warp;
  load_keys(unit);

  // logarithmic scaling of full-attention layers: query and bias times tau, each rounded to BF16 (the reference
  // multiplies in FP32 and casts back, my_inkling/model.py:583-590)
  const bool scaled = a.window == 0 && a.n_floor > 0;
  float tau = 1.f;
  if (scaled) tau = 1.f + a.alpha * logf(fmaxf((float)(position + 1) / (float)a.n_floor, 1.f));
  uint4 qf[kPieces];   // (loads that keep a place in L1: every warp of the block wants these rows. Seven sequences of 64 heads of 64 channels, 512 slots: 37.2 us past it, 36.5 so)
#pragma unroll
  for (int i = 0; i < kPieces; ++i) {
    qf[i] = g < n_heads ? reinterpret_cast<const uint4*>(a.q + ((size_t)b * a.heads + head0 + g) * C)[t + 4 * i] : make_uint4(0, 0, 0, 0);
    if (scaled) {
      qf[i].x = pack_bf16(bf16lo(qf[i].x) * tau, bf16hi(qf[i].x) * tau);
      qf[i].y = pack_bf16(bf16lo(qf[i].y) * tau, bf16hi(qf[i].y) * tau);
      qf[i].z = pack_bf16(bf16lo(qf[i].z) * tau, bf16hi(qf[i].z) * tau);
      qf[i].w = pack_bf16(bf16lo(qf[i].w) * tau, bf16hi(qf[i].w) * tau);
    }
  }
  const int rel_steps = (a.d_rel + 15) / 16, rel_pitch = rel_steps * 16;
  for (int i = tid; i < kAttnHeads * rel_pitch; i += kAttnThreads) {
    const int h = i / rel_pitch, j = i % rel_pitch;
    s_r[i] = (h < n_heads && j < a.d_rel) ? a.r[((size_t)b * a.heads + head0 + h) * a.d_rel + j] : (uint16_t)0;
  }
  __syncthreads();

  float acc[kHalves * 8][4];
#pragma unroll
  for (int i = 0; i < kHalves * 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
  float top = -INFINITY, total = 0.f;   // of head g over this warp's slots (total: this lane's slots only)
#pragma unroll 1
  for (; unit < unit1; unit += kAttnWarps) {
    const int slot0 = lo + unit * kAttnUnit;
    // ---- the values of the step are asked for before its scores are computed ...
    const uint4* vrow[4];
    bool vok[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int slot = slot0 + 2 * t + (i & 1) + (i >> 1) * 8;
      vok[i] = allowed_at(slot);   // (a slot that is not allowed may hold anything: it is not read)
      vrow[i] = reinterpret_cast<const uint4*>(slot == fresh_slot ? fresh_v : values + (size_t)slot * C);
    }
    constexpr int kAhead = kHalves > 2 ? 1 : kHalves;   // (256 channels: half of the row at a time, for the registers)
    uint4 vv[kAhead][4];
    auto load_values = [&](int h, uint4 (&to)[4]) {
#pragma unroll
      for (int i = 0; i < 4; ++i) to[i] = vok[i] ? ld_stream_16(vrow[i] + g + 8 * h) : make_uint4(0, 0, 0, 0);
    };
#pragma unroll
    for (int h = 0; h < kAhead; ++h) load_values(h, vv[h]);
    // ---- scores
    float sc[2][4];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      sc[n][0] = sc[n][1] = sc[n][2] = sc[n][3] = 0.f;
#pragma unroll
      for (int i = 0; i < kPieces; ++i) {
        mma_bf16(sc[n], qf[i].x, 0u, qf[i].y, 0u, kq[n][i].x, kq[n][i].y);
        mma_bf16(sc[n], qf[i].z, 0u, qf[i].w, 0u, kq[n][i].z, kq[n][i].w);
      }
    }
    // ---- ... and the next step's keys before the softmax
    load_keys(unit + kAttnWarps);
    float s[2][2];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      // relative bias of the step's slots: (r @ proj)[distance], a BF16 matmul (FP32 sum, rounded once)
      const int d_mine = distance_of(slot0 + n * 8 + g);
      const bool rel = slot0 + n * 8 + g < a.slots && d_mine >= 0 && d_mine < a.extent;
      float bias[4] = {0.f, 0.f, 0.f, 0.f};
      if (__any_sync(0xffffffffu, rel)) {
#pragma unroll 1
        for (int step = 0; step < rel_steps; ++step) {
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int j = step * 16 + 2 * t + (i & 1) + (i >> 1) * 8;
            w[i] = (rel && j < a.d_rel) ? (uint32_t)a.proj[(size_t)j * a.extent + d_mine] : 0u;
          }
          const uint32_t* r2 = reinterpret_cast<const uint32_t*>(s_r + g * rel_pitch + step * 16) + t;
          mma_bf16(bias, r2[0], 0u, r2[4], 0u, w[0] | (w[1] << 16), w[2] | (w[3] << 16));
        }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float add = round_bf16(bias[i]);
        if (scaled) add = round_bf16(add * tau);
        s[n][i] = allowed_at(slot0 + n * 8 + 2 * t + i) ? fmaf(sc[n][i], a.scale, add) : -INFINITY;
      }
    }
    float step_top = fmaxf(fmaxf(s[0][0], s[0][1]), fmaxf(s[1][0], s[1][1]));
    step_top = fmaxf(step_top, __shfl_xor_sync(0xffffffffu, step_top, 1));
    step_top = fmaxf(step_top, __shfl_xor_sync(0xffffffffu, step_top, 2));
    if (__any_sync(0xffffffffu, step_top > top)) {   // rare after the first steps: what has been summed moves to the new maximum
      const float next = fmaxf(top, step_top);
      const float factor = top == -INFINITY ? 0.f : __expf(top - next);
      top = next;
      total *= factor;
#pragma unroll
      for (int i = 0; i < kHalves * 8; ++i) {
        acc[i][0] *= factor;
        acc[i][1] *= factor;
        acc[i][2] *= factor;
        acc[i][3] *= factor;
      }
    }
    uint32_t p_hi[2], p_mid[2], p_lo[2];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const float p0 = s[n][0] == -INFINITY ? 0.f : __expf(s[n][0] - top), p1 = s[n][1] == -INFINITY ? 0.f : __expf(s[n][1] - top);
      total += p0 + p1;
      const float mid0 = p0 - bf16hi(__float_as_uint(p0)), mid1 = p1 - bf16hi(__float_as_uint(p1));
      const float lo0 = mid0 - bf16hi(__float_as_uint(mid0)), lo1 = mid1 - bf16hi(__float_as_uint(mid1));
      constexpr float kNext = 0x1p-40f;
      p_hi[n] = high_halves(p0, p1);
      p_mid[n] = high_halves(fmaxf(mid0, p0 * kNext), fmaxf(mid1, p1 * kNext));
      p_lo[n] = high_halves(0.5f * fmaxf(lo0, p0 * kNext), 0.5f * fmaxf(lo1, p1 * kNext));
    }
    // ---- weighted values: 8 channels of the lane's piece, one instruction each
#pragma unroll
    for (int h = 0; h < kHalves; ++h) {
      uint4(&v4)[4] = vv[h < kAhead ? h : 0];
      if (h >= kAhead) load_values(h, v4);
      const uint32_t w0[4] = {v4[0].x, v4[0].y, v4[0].z, v4[0].w}, w1[4] = {v4[1].x, v4[1].y, v4[1].z, v4[1].w};
      const uint32_t w2[4] = {v4[2].x, v4[2].y, v4[2].z, v4[2].w}, w3[4] = {v4[3].x, v4[3].y, v4[3].z, v4[3].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int odd = 0; odd < 2; ++odd) {
          const uint32_t b0 = __byte_perm(w0[j], w1[j], odd ? 0x7632 : 0x5410), b1 = __byte_perm(w2[j], w3[j], odd ? 0x7632 : 0x5410);
          mma_bf16(acc[h * 8 + 2 * j + odd], p_hi[0], p_mid[0], p_hi[1], p_mid[1], b0, b1);
          mma_bf16(acc[h * 8 + 2 * j + odd], p_lo[0], p_lo[0], p_lo[1], p_lo[1], b0, b1);   // (a half of lo in either row)
        }
      }
    }
  }
  total += __shfl_xor_sync(0xffffffffu, total, 1);
  total += __shfl_xor_sync(0xffffffffu, total, 2);
  __syncthreads();   // (the relative states make room)
  // ---- the warps' sums, then the block's: thread = (head, channels)
  {
    float* mine = s_acc + (warp * kAttnHeads + g) * (C + 2);
    if (t == 0) {
      mine[C] = top;
      mine[C + 1] = total;
    }
#pragma unroll
    for (int h = 0; h < kHalves; ++h)
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int j = 0; j < 8; ++j) mine[h * 64 + 16 * t + 8 * n + j] = acc[h * 8 + j][n] + acc[h * 8 + j][2 + n];
  }
  __syncthreads();
  constexpr int kPairs = C / 2;                       // channel pairs of a head
  const int stride = kAttnPartial + C;
  for (int i = tid; i < n_heads * kPairs; i += kAttnThreads) {
    const int h = i / kPairs, pair = i % kPairs;
    float all_top = -INFINITY;
#pragma unroll
    for (int w = 0; w < kAttnWarps; ++w) all_top = fmaxf(all_top, s_acc[(w * kAttnHeads + h) * (C + 2) + C]);
    float o0 = 0.f, o1 = 0.f, sum = 0.f;
#pragma unroll
    for (int w = 0; w < kAttnWarps; ++w) {
      const float* from = s_acc + (w * kAttnHeads + h) * (C + 2);
      const float weight = from[C] == -INFINITY ? 0.f : __expf(from[C] - all_top);
      o0 = fmaf(from[2 * pair], weight, o0);
      o1 = fmaf(from[2 * pair + 1], weight, o1);
      sum = fmaf(from[C + 1], weight, sum);
    }
    const size_t row = (size_t)b * a.heads + head0 + h;
    if (a.splits == 1) {
      const float inv = 1.f / sum;
      reinterpret_cast<uint32_t*>(a.out + row * C)[pair] = pack_bf16(o0 * inv, o1 * inv);
    } else if (CLUSTER) {
      float* mine = s_block + h * (C + 2);
      if (pair == 0) *reinterpret_cast<float2*>(mine + C) = make_float2(all_top, sum);
      *reinterpret_cast<float2*>(mine + 2 * pair) = make_float2(o0, o1);
    } else {
      float* mine = a.partial + (row * a.splits + split) * stride;
      if (pair == 0) *reinterpret_cast<float2*>(mine) = make_float2(all_top, sum);
      *reinterpret_cast<float2*>(mine + kAttnPartial + 2 * pair) = make_float2(o0, o1);
    }
  }
  if (a.splits == 1) return;
  //   out = sum_i acc_i e^(m_i - M) / sum_i l_i e^(m_i - M)
  if constexpr (CLUSTER) {
    cluster_sync();
    for (int i = split * kAttnThreads + tid; i < n_heads * kPairs; i += a.splits * kAttnThreads) {
      const int h = i / kPairs, pair = i % kPairs;
      float2 head[kAttnCluster], val[kAttnCluster];
      float all_top = -INFINITY;
#pragma unroll
      for (int s = 0; s < kAttnCluster; ++s) {
        head[s] = s < a.splits ? ld_cluster_float2(s_block + h * (C + 2) + C, s) : make_float2(-INFINITY, 0.f);
        val[s] = s < a.splits ? ld_cluster_float2(s_block + h * (C + 2) + 2 * pair, s) : make_float2(0.f, 0.f);
        all_top = fmaxf(all_top, head[s].x);
      }
      float o0 = 0.f, o1 = 0.f, sum = 0.f;
#pragma unroll
      for (int s = 0; s < kAttnCluster; ++s) {
        const float weight = head[s].x == -INFINITY ? 0.f : __expf(head[s].x - all_top);
        sum = fmaf(head[s].y, weight, sum);
        o0 = fmaf(val[s].x, weight, o0);
        o1 = fmaf(val[s].y, weight, o1);
      }
      const float inv = 1.f / sum;
      reinterpret_cast<uint32_t*>(a.out + ((size_t)b * a.heads + head0 + h) * C)[pair] = pack_bf16(o0 * inv, o1 * inv);
    }
    cluster_sync();   // (a block's sums stay until everybody has read them)
    return;
  }
  // The block that stores the last partial of its heads joins them all.
  __threadfence();   // every writer pushes its own stores out before the block is counted
  __syncthreads();
  if (tid == 0) {
    unsigned* arrived = a.arrived + (size_t)b * gridDim.y + blockIdx.y;
    s_last = atomicAdd(arrived, 1u) + 1u == (unsigned)a.splits;
    if (s_last) *arrived = 0u;   // left as found, for the next launch
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // first every part's weight, all parts at once: [head][part]; then the sums, sixteen parts in flight
  float* s_weight = s_acc;
  float* s_inv = s_acc + kAttnHeads * kAttnMaxSplits;
  for (int h = warp; h < n_heads; h += kAttnWarps) {
    const float* base = a.partial + ((size_t)b * a.heads + head0 + h) * a.splits * stride;
    constexpr int kPerLane = kAttnMaxSplits / 32;
    float2 head[kPerLane];
    float all_top = -INFINITY, sum = 0.f;
#pragma unroll
    for (int n = 0; n < kPerLane; ++n) {
      const int s = n * 32 + lane;
      head[n] = s < a.splits ? __ldcg(reinterpret_cast<const float2*>(base + (size_t)s * stride)) : make_float2(-INFINITY, 0.f);
      all_top = fmaxf(all_top, head[n].x);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) all_top = fmaxf(all_top, __shfl_xor_sync(0xffffffffu, all_top, o));
#pragma unroll
    for (int n = 0; n < kPerLane; ++n) {
      const float weight = head[n].x == -INFINITY ? 0.f : __expf(head[n].x - all_top);
      s_weight[h * kAttnMaxSplits + n * 32 + lane] = weight;
      sum = fmaf(head[n].y, weight, sum);
    }
    sum = warp_sum(sum);
    if (lane == 0) s_inv[h] = 1.f / sum;
  }
  __syncthreads();
  for (int i = tid; i < n_heads * (C / 4); i += kAttnThreads) {
    const int h = i / (C / 4), quad = i % (C / 4);
    const size_t row = (size_t)b * a.heads + head0 + h;
    const float* base = a.partial + row * a.splits * stride + kAttnPartial + 4 * quad;
    const float* weights = s_weight + h * kAttnMaxSplits;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int s0 = 0; s0 < a.splits; s0 += 16) {
      float4 v[16];
#pragma unroll
      for (int n = 0; n < 16; ++n) v[n] = s0 + n < a.splits ? __ldcg(reinterpret_cast<const float4*>(base + (size_t)(s0 + n) * stride)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int n = 0; n < 16; ++n) {
        const float weight = weights[s0 + n];   // (zero beyond the last part)
        o.x = fmaf(v[n].x, weight, o.x);
        o.y = fmaf(v[n].y, weight, o.y);
        o.z = fmaf(v[n].z, weight, o.z);
        o.w = fmaf(v[n].w, weight, o.w);
      }
    }
    const float inv = s_inv[h];
    reinterpret_cast<uint2*>(a.out + row * C)[quad] = make_uint2(pack_bf16(o.x * inv, o.y * inv), pack_bf16(o.z * inv, o.w * inv));
  }
}

// The form for small problems, where all parts are resident at once and latency counts: one block per (64 slots, group of
// up to eight heads of one key/value head, sequence), on the CUDA cores in FP32. Every thread asks for its share of the key
// rows and value rows at once (which slots are allowed is known before any score) and keeps them for all heads of the
// group; with one block per head, as before, eight blocks read the same rows and the join of a head waited for eight times as
// many of them. The order of all sums is that of one block per head, so the results are the same bits: a decode step of
// several layers turns any last-bit difference into another routing weight, another rounding, and so on.
constexpr int kSmallThreads = 256;
constexpr int kSmallMostBlocks = 148 * 4;
constexpr int kSmallKeys = 8;                                        // slots a warp scores
constexpr int kSmallSlots = kSmallThreads / 32 * kSmallKeys;         // slots per block: 64

template <int C, bool CLUSTER>
__global__ void __launch_bounds__(kSmallThreads) decode_attention_small_kernel(AttnArgs a) {
  constexpr int kWords = C / 2;                          // 32-bit words of a row = channel pairs
  constexpr int kPerLane = (kWords + 31) / 32;           // words of a key row per lane
  constexpr int kParts = kSmallThreads / kWords;         // threads per channel pair in the value pass
  constexpr int kValues = kSmallSlots / kParts;          // value rows per thread
  static_assert(kSmallThreads % kWords == 0 && kSmallSlots % kParts == 0, "head_dim does not tile the block");
  extern __shared__ __align__(16) unsigned char s_raw[];
  float2* s_part = reinterpret_cast<float2*>(s_raw);                                // [heads][parts][pairs]
  float* s_q = reinterpret_cast<float*>(s_part + kAttnHeads * kSmallThreads);       // [heads][C]
  float* s_scores = s_q + kAttnHeads * C;                                           // [heads][64]: biases, scores, exponentials
  float* s_sum = s_scores + kAttnHeads * kSmallSlots;                               // [heads][parts]
  float* s_block = s_sum + kAttnHeads * kParts;                                     // [heads][C + 2]: this block's sums, for its cluster
  uint16_t* s_r = reinterpret_cast<uint16_t*>(s_block + kAttnHeads * (C + 2));      // [heads][d_rel]
  __shared__ float s_top[kAttnHeads];
  __shared__ bool s_last;
  pdl_wait();
  pdl_trigger();
  const int split = blockIdx.x, b = blockIdx.z, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int group = a.heads / a.kv_heads, chunks = (group + kAttnHeads - 1) / kAttnHeads;
  const int kv_head = blockIdx.y / chunks, chunk = blockIdx.y % chunks;
  const int head0 = kv_head * group + chunk * kAttnHeads, n_heads = min(kAttnHeads, group - chunk * kAttnHeads);
  const int slot_base = split * kSmallSlots;
  const size_t row0 = ((size_t)b * a.kv_heads + kv_head) * a.slots;
  const uint16_t* keys = a.k + row0 * C;
  const uint16_t* values = a.v + row0 * C;
  const uint16_t* fresh_k = a.new_k ? a.new_k + ((size_t)b * a.kv_heads + kv_head) * C : nullptr;
  const uint16_t* fresh_v = a.new_k ? a.new_v + ((size_t)b * a.kv_heads + kv_head) * C : nullptr;
  const int pair = tid % kWords, part = tid / kWords;   // value pass: this thread's channel pair, its slots part, part + kParts, ...
  // All rows of the block are asked for before the position is known (a short cache is mostly in use); what turns out not
  // to be allowed is dropped below. In a long one that would read far beyond the position: there the position comes first.
  constexpr bool kEarly = CLUSTER;
  uint32_t kw[kSmallKeys][kPerLane], vw[kValues];
  if (kEarly) {
#pragma unroll
    for (int j = 0; j < kSmallKeys; ++j) {
      const int slot = slot_base + warp * kSmallKeys + j;
      const uint32_t* row = reinterpret_cast<const uint32_t*>(keys + (size_t)slot * C);
#pragma unroll
      for (int i = 0; i < kPerLane; ++i) kw[j][i] = (slot < a.slots && i * 32 + lane < kWords) ? __ldcg(row + i * 32 + lane) : 0u;
    }
#pragma unroll
    for (int n = 0; n < kValues; ++n) {
      const int slot = slot_base + part + n * kParts;
      vw[n] = slot < a.slots ? __ldcg(reinterpret_cast<const uint32_t*>(values + (size_t)slot * C) + pair) : 0u;
    }
  }
  const int position = (int)*a.position;
  const int reach = position - (int)(a.pad_counts ? a.pad_counts[b] : 0);
  const int ring_position = a.window ? position % a.window : 0;
  auto distance_of = [&](int slot) -> int {
    if (!a.window) return position - slot;
    const int d = ring_position - (slot < a.window ? slot : slot % a.window);
    return d < 0 ? d + a.window : d;
  };
  auto allowed_at = [&](int slot) -> bool {
    const int d = distance_of(slot);
    return slot < a.slots && d >= 0 && d <= reach;
  };
  // parts beyond the position have nothing to add (in a full layer; a ring's slots beyond it are masked one by one)
  const int active = a.window || position + 1 >= a.slots ? a.splits : position / kSmallSlots + 1;
  if (!CLUSTER && split >= active) return;
  const int fresh_slot = a.new_k ? (a.window ? ring_position : position) : -1;
  const bool fresh_here = fresh_slot >= slot_base && fresh_slot < slot_base + kSmallSlots && fresh_slot < a.slots;
  bool k_allowed[kSmallKeys];
#pragma unroll
  for (int j = 0; j < kSmallKeys; ++j) {
    const int slot = slot_base + warp * kSmallKeys + j;
    k_allowed[j] = allowed_at(slot);
    if (!kEarly || (fresh_here && slot == fresh_slot)) {
      const uint32_t* row = reinterpret_cast<const uint32_t*>(slot == fresh_slot ? fresh_k : keys + (size_t)slot * C);
#pragma unroll
      for (int i = 0; i < kPerLane; ++i) kw[j][i] = (k_allowed[j] && i * 32 + lane < kWords) ? __ldcg(row + i * 32 + lane) : 0u;
    }
  }
#pragma unroll
  for (int n = 0; n < kValues; ++n) {
    const int slot = slot_base + part + n * kParts;
    const bool ok = allowed_at(slot);   // (a slot that is not allowed may hold anything: it does not count)
    if (!kEarly || (fresh_here && slot == fresh_slot))
      vw[n] = ok ? __ldcg(reinterpret_cast<const uint32_t*>(slot == fresh_slot ? fresh_v : values + (size_t)slot * C) + pair) : 0u;
    else if (!ok) vw[n] = 0u;
  }
  if (a.new_k && chunk == 0 && fresh_here && tid < kWords) {
    reinterpret_cast<uint32_t*>(a.k_store + (row0 + fresh_slot) * C)[tid] = __ldcg(reinterpret_cast<const uint32_t*>(fresh_k) + tid);
    reinterpret_cast<uint32_t*>(a.v_store + (row0 + fresh_slot) * C)[tid] = __ldcg(reinterpret_cast<const uint32_t*>(fresh_v) + tid);
  }
  const bool scaled = a.window == 0 && a.n_floor > 0;
  float tau = 1.f;
  if (scaled) tau = 1.f + a.alpha * logf(fmaxf((float)(position + 1) / (float)a.n_floor, 1.f));
  for (int i = tid; i < n_heads * C; i += kSmallThreads) {
    const float x = bf16_to_f32(a.q[((size_t)b * a.heads + head0) * C + i]);
    s_q[i] = scaled ? round_bf16(x * tau) : x;
  }
  for (int i = tid; i < n_heads * a.d_rel; i += kSmallThreads) s_r[i] = a.r[((size_t)b * a.heads + head0) * a.d_rel + i];
  __syncthreads();
  // relative bias of this block's slots: (r @ proj)[distance], a BF16 matmul (FP32 sum, rounded once)
  {
    const int slot = slot_base + tid % kSmallSlots, d = distance_of(slot);
    constexpr int kStep = kSmallThreads / kSmallSlots, kMine = kAttnHeads / kStep;   // heads h0, h0 + 4
    const int h0 = tid / kSmallSlots;
    float sum[kMine];
#pragma unroll
    for (int n = 0; n < kMine; ++n) sum[n] = 0.f;
    const bool rel = slot < a.slots && d >= 0 && d < a.extent;
    if (rel) {
      // (sixteen patterns in one round trip; eight at a time the calls of one round took up to 4 % more: seven sequences of 64 heads on 8, 256
      // channels, 128 slots 14.2 us, 13.8 so; one of 16 on 16, 128 channels, 512 slots 8.4 / 8.2)
#pragma unroll 16
      for (int j = 0; j < a.d_rel; ++j) {
        const float p = bf16_to_f32(a.proj[(size_t)j * a.extent + d]);
#pragma unroll
        for (int n = 0; n < kMine; ++n)
          if (h0 + n * kStep < n_heads) sum[n] = fmaf(bf16_to_f32(s_r[(h0 + n * kStep) * a.d_rel + j]), p, sum[n]);
      }
    }
#pragma unroll
    for (int n = 0; n < kMine; ++n) {
      float bias = 0.f;
      if (rel) {
        bias = round_bf16(sum[n]);
        if (scaled) bias = round_bf16(bias * tau);
      }
      s_scores[(h0 + n * kStep) * kSmallSlots + tid % kSmallSlots] = bias;
    }
  }
  __syncthreads();
  // ---- scores: warp w holds the key rows of the slots w * 8 .. w * 8 + 7 of the block
  bool mine_allowed = false;   // of the slot this lane ends up with
  const int mine = reduced_row<kSmallKeys>(lane);
#pragma unroll
  for (int j = 0; j < kSmallKeys; ++j) mine_allowed = j == mine ? k_allowed[j] : mine_allowed;
#pragma unroll 4
  for (int h = 0; h < n_heads; ++h) {
    float dot[kSmallKeys];
    float2 q2[kPerLane];
#pragma unroll
    for (int i = 0; i < kPerLane; ++i) q2[i] = i * 32 + lane < kWords ? reinterpret_cast<const float2*>(s_q + h * C)[i * 32 + lane] : make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < kSmallKeys; ++j) {
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < kPerLane; ++i) {
        if (i * 32 + lane < kWords) {
          sum = fmaf(q2[i].x, bf16lo(kw[j][i]), sum);
          sum = fmaf(q2[i].y, bf16hi(kw[j][i]), sum);
        }
      }
      dot[j] = sum;
    }
    const float total = multi_reduce<kSmallKeys>(dot, lane);
    if (reduced_owner<kSmallKeys>(lane)) {
      float* at = s_scores + h * kSmallSlots + warp * kSmallKeys + mine;
      *at = mine_allowed ? total * a.scale + *at : -INFINITY;
    }
  }
  __syncthreads();
  // ---- a warp per head: the maximum of its 64 scores, then the exponentials
  for (int h = warp; h < n_heads; h += kSmallThreads / 32) {
    float* sc = s_scores + h * kSmallSlots;
    const float s0 = sc[lane], s1 = sc[lane + 32];
    float top = fmaxf(s0, s1);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    sc[lane] = (s0 == -INFINITY) ? 0.f : __expf(s0 - top);
    sc[lane + 32] = (s1 == -INFINITY) ? 0.f : __expf(s1 - top);
    if (lane == 0) s_top[h] = top;
  }
  __syncthreads();
#pragma unroll 4
  for (int h = 0; h < n_heads; ++h) {
    float acc0 = 0.f, acc1 = 0.f, sum = 0.f;
#pragma unroll
    for (int n = 0; n < kValues; ++n) {
      const float p = s_scores[h * kSmallSlots + part + n * kParts];
      acc0 = fmaf(p, bf16lo(vw[n]), acc0);
      acc1 = fmaf(p, bf16hi(vw[n]), acc1);
      sum += p;
    }
    s_part[h * kSmallThreads + tid] = make_float2(acc0, acc1);
    if (pair == 0) s_sum[h * kParts + part] = sum;
  }
  __syncthreads();
  const int stride = kAttnPartial + C;
  for (int i = tid; i < n_heads * kWords; i += kSmallThreads) {
    const int h = i / kWords, w = i % kWords;
    float o0 = 0.f, o1 = 0.f, total = 0.f;
#pragma unroll
    for (int p = 0; p < kParts; ++p) {
      const float2 v = s_part[h * kSmallThreads + p * kWords + w];
      o0 += v.x;
      o1 += v.y;
      total += s_sum[h * kParts + p];
    }
    const size_t row = (size_t)b * a.heads + head0 + h;
    if (a.splits == 1) {
      const float inv = 1.f / total;
      reinterpret_cast<uint32_t*>(a.out + row * C)[w] = f32_to_bf16_bits(o0 * inv) | (f32_to_bf16_bits(o1 * inv) << 16);
    } else {
      float* to = CLUSTER ? s_block + h * (C + 2) + 2 * w : a.partial + (row * a.splits + split) * stride + kAttnPartial + 2 * w;
      *reinterpret_cast<float2*>(to) = make_float2(o0, o1);
      if (w == 0) *reinterpret_cast<float2*>(CLUSTER ? s_block + h * (C + 2) + C : a.partial + (row * a.splits + split) * stride) = make_float2(s_top[h], total);
    }
  }
  if (a.splits == 1) return;
  // ---- join: part p of the sum takes every kParts-th partial, then the parts are added up
  if constexpr (CLUSTER) {
    cluster_sync();
    for (int i = split * kSmallThreads + tid; i < n_heads * kWords; i += a.splits * kSmallThreads) {
      const int h = i / kWords, w = i % kWords;
      float2 head[kAttnCluster], val[kAttnCluster];
      float all_top = -INFINITY;
#pragma unroll
      for (int s = 0; s < kAttnCluster; ++s) {
        head[s] = s < a.splits ? ld_cluster_float2(s_block + h * (C + 2) + C, s) : make_float2(-INFINITY, 0.f);
        val[s] = s < a.splits ? ld_cluster_float2(s_block + h * (C + 2) + 2 * w, s) : make_float2(0.f, 0.f);
        all_top = fmaxf(all_top, head[s].x);
      }
      float f0 = 0.f, f1 = 0.f, sum_all = 0.f;
#pragma unroll
      for (int p = 0; p < kParts; ++p) {
        float o0 = 0.f, o1 = 0.f, total = 0.f;
#pragma unroll
        for (int s = p; s < kAttnCluster; s += kParts) {
          if (head[s].x == -INFINITY) continue;
          const float weight = __expf(head[s].x - all_top);
          total = fmaf(head[s].y, weight, total);
          o0 = fmaf(val[s].x, weight, o0);
          o1 = fmaf(val[s].y, weight, o1);
        }
        f0 += o0;
        f1 += o1;
        sum_all += total;
      }
      const float inv = 1.f / sum_all;
      reinterpret_cast<uint32_t*>(a.out + ((size_t)b * a.heads + head0 + h) * C)[w] = f32_to_bf16_bits(f0 * inv) | (f32_to_bf16_bits(f1 * inv) << 16);
    }
    cluster_sync();   // (a block's sums stay until everybody has read them)
  } else {
    __threadfence();   // every writer pushes its own stores out before the block is counted
    __syncthreads();
    if (tid == 0) {
      unsigned* arrived = a.arrived + (size_t)b * gridDim.y + blockIdx.y;
      s_last = atomicAdd(arrived, 1u) + 1u == (unsigned)active;
      if (s_last) *arrived = 0u;   // left as found, for the next launch
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // a warp per head: every partial's weight (zero beyond the active ones and for empty ones) and their total
    float* s_weight = s_q;   // [heads][64]
    for (int h = warp; h < n_heads; h += kSmallThreads / 32) {
      const float* base = a.partial + ((size_t)b * a.heads + head0 + h) * a.splits * stride;
      constexpr int kEach = kAttnMaxSplits / 32;
      float2 head[kEach];
      float all_top = -INFINITY;
#pragma unroll
      for (int n = 0; n < kEach; ++n) {
        const int s = n * 32 + lane;
        head[n] = s < active ? __ldcg(reinterpret_cast<const float2*>(base + (size_t)s * stride)) : make_float2(-INFINITY, 0.f);
        all_top = fmaxf(all_top, head[n].x);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) all_top = fmaxf(all_top, __shfl_xor_sync(0xffffffffu, all_top, o));
#pragma unroll
      for (int n = 0; n < kEach; ++n) {
        s_weight[h * kAttnMaxSplits + n * 32 + lane] = head[n].x == -INFINITY ? 0.f : __expf(head[n].x - all_top);
        s_scores[h * kAttnMaxSplits + n * 32 + lane] = head[n].y;
      }
    }
    __syncthreads();
    constexpr int kMost = kAttnMaxSplits / kParts;   // partials per thread and head
#pragma unroll 1
    for (int h = 0; h < n_heads; ++h) {
      const float* base = a.partial + ((size_t)b * a.heads + head0 + h) * a.splits * stride + kAttnPartial + 2 * pair;
      float2 v[kMost];
#pragma unroll
      for (int n = 0; n < kMost; ++n) v[n] = part + n * kParts < active ? __ldcg(reinterpret_cast<const float2*>(base + (size_t)(part + n * kParts) * stride)) : make_float2(0.f, 0.f);
      float o0 = 0.f, o1 = 0.f, total = 0.f;
#pragma unroll
      for (int n = 0; n < kMost; ++n) {   // (an empty partial's weight is zero and its sums are zero: nothing changes)
        const float weight = s_weight[h * kAttnMaxSplits + part + n * kParts];
        total = fmaf(s_scores[h * kAttnMaxSplits + part + n * kParts], weight, total);
        o0 = fmaf(v[n].x, weight, o0);
        o1 = fmaf(v[n].y, weight, o1);
      }
      s_part[h * kSmallThreads + tid] = make_float2(o0, o1);
      if (pair == 0) s_sum[h * kParts + part] = total;
    }
    __syncthreads();
    for (int i = tid; i < n_heads * kWords; i += kSmallThreads) {
      const int h = i / kWords, w = i % kWords;
      float f0 = 0.f, f1 = 0.f, sum_all = 0.f;
#pragma unroll
      for (int p = 0; p < kParts; ++p) {
        const float2 v = s_part[h * kSmallThreads + p * kWords + w];
        f0 += v.x;
        f1 += v.y;
        sum_all += s_sum[h * kParts + p];
      }
      const float inv = 1.f / sum_all;
      reinterpret_cast<uint32_t*>(a.out + ((size_t)b * a.heads + head0 + h) * C)[w] = f32_to_bf16_bits(f0 * inv) | (f32_to_bf16_bits(f1 * inv) << 16);
    }
  }
}

// the new token's key and value into slot `position` (modulo the window in a sliding layer) of both caches
__global__ void update_kv_kernel(const uint16_t* __restrict__ new_k, const uint16_t* __restrict__ new_v,
                                 uint16_t* __restrict__ k_cache, uint16_t* __restrict__ v_cache,
                                 const int64_t* __restrict__ position, int c, int slots, int window) {
  const long long p = *position;
  const long long slot = window ? p % window : p;
  if (slot < 0 || slot >= slots) return;   // a full cache: nothing is written (the host-side check reports it)
  const size_t row = blockIdx.x;           // (sequence, kv head)
  for (int i = threadIdx.x; i < c; i += blockDim.x) {
    k_cache[(row * slots + slot) * c + i] = new_k[row * c + i];
    v_cache[(row * slots + slot) * c + i] = new_v[row * c + i];
  }
}

}  // namespace ink

using namespace ink;

static size_t attention_counter_bytes(int batch, int heads) { return ((size_t)batch * heads * sizeof(unsigned) + 255) / 256 * 256; }
extern "C" size_t ink_decode_attention_counter_bytes(int batch, int heads) { return attention_counter_bytes(batch, heads); }

// Splits along the cache at most: what the workspace is sized for, whatever the number of key/value heads. (Up to
// kAttnCluster parts always meet in a cluster and need none.)
static int attention_max_splits(int slots) {
  const int whole = (slots + kAttnMinSlots - 1) / kAttnMinSlots;
  return whole < kAttnMaxSplits ? whole : kAttnMaxSplits;
}

// Where all 64-slot parts are resident at once the small form takes them. Else the number of parts that takes the fewest
// rounds of (steps a warp makes + what a block costs beside, about four steps' time), a round being what is resident at once.
static int attention_splits(int batch, int kv_heads, int chunks, int head_dim, int slots, bool* small) {
  const int pairs = batch * kv_heads * chunks, whole = (slots + kAttnMinSlots - 1) / kAttnMinSlots;
  *small = whole <= kAttnMaxSplits && (long long)whole * pairs <= kSmallMostBlocks;
  int splits = whole, best = 0x7fffffff;
  for (int n = 1, most = attention_max_splits(slots); n <= most && !*small; ++n) {
    const bool cluster = n > 1 && n <= kAttnCluster;
    const long long resident = cluster ? kAttnClusters[head_dim > 128][n] : kAttnSms * kAttnPerSm(head_dim);
    const long long wanted = cluster ? pairs : (long long)pairs * n, cost = (wanted + resident - 1) / resident * (4 + (whole + n - 1) / n);
    if (cost <= best) {   // (of equals the finer: sequences may be shorter than the cache)
      best = (int)cost;
      splits = n;
    }
  }
  return splits;
}

extern "C" int ink_decode_attention_joins(int batch, int heads, int kv_heads, int head_dim, int slots) {
  if (batch <= 0 || kv_heads <= 0 || heads <= 0 || slots <= 0) return 0;
  bool small;
  return attention_splits(batch, kv_heads, (heads / kv_heads + kAttnHeads - 1) / kAttnHeads, head_dim, slots, &small) > kAttnCluster;
}

extern "C" size_t ink_decode_attention_workspace_bytes(int batch, int heads, int head_dim, int slots) {
  const size_t splits = (size_t)attention_max_splits(slots);
  return splits <= kAttnCluster ? 0 : attention_counter_bytes(batch, heads) + sizeof(float) * (size_t)batch * heads * splits * (kAttnPartial + head_dim);
}

template <int C>
static int launch_decode_attention(const AttnArgs& a, bool small, dim3 grid, cudaStream_t stream) {
  const size_t sums = sizeof(float) * kAttnWarps * kAttnHeads * (C + 2), rel = sizeof(uint16_t) * kAttnHeads * ((size_t)(a.d_rel + 15) / 16 * 16);
  static_assert(kAttnWarps * (C + 2) > kAttnMaxSplits + 1, "the join's weights fit where the warps' sums were");
  const size_t smem_small = sizeof(float) * kAttnHeads * (2 * kSmallThreads + C + kSmallSlots + kSmallThreads / (C / 2) + C + 2) + rel;
  const size_t smem = small ? smem_small : sums > rel ? sums : rel;
  static_assert(kSmallSlots == kAttnMaxSplits && C >= kAttnMaxSplits, "the join's weights fit where queries and scores were");
  INK_REQUIRE(rel <= 160 * 1024, kUnsupportedShape, "decode_attention: d_rel=%d is too wide", a.d_rel);
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = dim3(small ? kSmallThreads : kAttnThreads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[0].val.programmaticStreamSerializationAllowed = 1;
  attributes[1].id = cudaLaunchAttributeClusterDimension;
  attributes[1].val.clusterDim.x = grid.x;
  attributes[1].val.clusterDim.y = attributes[1].val.clusterDim.z = 1;
  const bool cluster = a.splits > 1 && a.splits <= kAttnCluster;
  // Clusters may start while the kernel in front still runs, which saves a call 1 to 2 us, unless they hardly all fit: those that
  // find an SM still taken would make a second round (seven sequences of 64 heads on 8 at 3 000 slots, 56 clusters of seven where 56
  // fit: 45 us in a layer, 29 so). Nor do the other forms, whose grids fill the chip: their blocks would take
  // the places unevenly (50.1 us for 46.7, seven sequences of 32 heads on 32, 256 channels, 512 slots).
  const int fit = cluster ? kAttnClusters[C > 128][a.splits] : 0;
  const bool early = cluster && (small || (long long)grid.y * grid.z <= fit - fit / 16);
  config.attrs = early ? attributes : attributes + 1;
  config.numAttrs = cluster ? (early ? 2 : 1) : 0;
  void (*kernel)(AttnArgs) = small ? (cluster ? decode_attention_small_kernel<C, true> : decode_attention_small_kernel<C, false>)
                                   : (cluster ? decode_attention_kernel<C, true> : decode_attention_kernel<C, false>);
  if (smem > 40 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const cudaError_t e = cudaLaunchKernelEx(&config, kernel, a);
  INK_REQUIRE(e == cudaSuccess, kLaunchFailed, "decode_attention: launch failed: %s", cudaGetErrorString(e));
  return kOk;
}

extern "C" int ink_decode_attention(const void* q, const void* r, const void* proj, void* k_cache,
                                    void* v_cache, const int64_t* position, const int64_t* pad_counts, void* out,
                                    int batch, int heads, int kv_heads, int head_dim, int d_rel, int rel_extent, int slots,
                                    int window, int n_floor, float alpha, float scale, const void* new_k,
                                    const void* new_v, void* workspace, size_t workspace_bytes, ink_stream_t stream) {
  INK_REQUIRE(q && r && proj && k_cache && v_cache && position && out, kBadArgument, "decode_attention: null pointer argument");
  INK_REQUIRE(batch >= 0 && heads > 0 && kv_heads > 0 && heads % kv_heads == 0, kBadArgument,
              "decode_attention: batch=%d heads=%d kv_heads=%d", batch, heads, kv_heads);
  INK_REQUIRE(head_dim == 64 || head_dim == 128 || head_dim == 256, kUnsupportedShape,
              "decode_attention: head_dim=%d unsupported (built for 64, 128 and 256)", head_dim);
  INK_REQUIRE(d_rel > 0 && rel_extent > 0 && slots > 0 && window >= 0 && (window == 0 || window <= slots), kBadArgument,
              "decode_attention: d_rel=%d rel_extent=%d slots=%d window=%d", d_rel, rel_extent, slots, window);
  INK_REQUIRE((new_k == nullptr) == (new_v == nullptr), kBadArgument, "decode_attention: new_k and new_v come together");
  const int group = heads / kv_heads, chunks = (group + kAttnHeads - 1) / kAttnHeads;
  INK_REQUIRE((long long)kv_heads * chunks <= 65535 && batch <= 65535, kUnsupportedShape,
              "decode_attention: %d heads or %d sequences exceed the grid", heads, batch);
  const size_t need = ink_decode_attention_workspace_bytes(batch, heads, head_dim, slots);
  INK_REQUIRE(need == 0 || (workspace && workspace_bytes >= need), kBadArgument,
              "decode_attention: workspace of %zu bytes needed, %zu given", need, workspace_bytes);
  INK_REQUIRE(aligned16(q) && aligned16(k_cache) && aligned16(v_cache) && aligned16(out) &&
                  (need == 0 || aligned16(workspace)),
              kMisaligned, "decode_attention: buffers must be 16-byte aligned");
  if (batch == 0) return kOk;
  if (!aligned16(new_k) || !aligned16(new_v)) {   // (the kernels read these rows 16 bytes at a time: stored first instead)
    if (int rc = ink_update_kv(new_k, new_v, k_cache, v_cache, position, batch, kv_heads, head_dim, slots, window, stream)) return rc;
    new_k = new_v = nullptr;
  }
  bool small;
  const int splits = attention_splits(batch, kv_heads, chunks, head_dim, slots, &small);
  AttnArgs a{(const uint16_t*)q, (const uint16_t*)r, (const uint16_t*)proj, (const uint16_t*)k_cache, (const uint16_t*)v_cache,
             position, pad_counts, (const uint16_t*)new_k, (const uint16_t*)new_v, (uint16_t*)k_cache, (uint16_t*)v_cache,
             (float*)((char*)workspace + attention_counter_bytes(batch, heads)), (unsigned*)workspace, (uint16_t*)out, heads, kv_heads,
             d_rel, rel_extent, slots, window, n_floor, splits, alpha, scale};
  const dim3 grid((unsigned)splits, (unsigned)(kv_heads * chunks), (unsigned)batch);
  if (head_dim == 64) return launch_decode_attention<64>(a, small, grid, (cudaStream_t)stream);
  if (head_dim == 128) return launch_decode_attention<128>(a, small, grid, (cudaStream_t)stream);
  return launch_decode_attention<256>(a, small, grid, (cudaStream_t)stream);
}

extern "C" int ink_update_kv(const void* new_k, const void* new_v, void* k_cache, void* v_cache, const int64_t* position,
                             int batch, int kv_heads, int head_dim, int slots, int window, ink_stream_t stream) {
  INK_REQUIRE(new_k && new_v && k_cache && v_cache && position, kBadArgument, "update_kv: null pointer argument");
  INK_REQUIRE(batch >= 0 && kv_heads > 0 && head_dim > 0 && slots > 0 && window >= 0 && (window == 0 || window <= slots),
              kBadArgument, "update_kv: batch=%d kv_heads=%d head_dim=%d slots=%d window=%d", batch, kv_heads, head_dim, slots, window);
  if (batch == 0) return kOk;
  update_kv_kernel<<<batch * kv_heads, 128, 0, (cudaStream_t)stream>>>((const uint16_t*)new_k, (const uint16_t*)new_v,
                                                                       (uint16_t*)k_cache, (uint16_t*)v_cache, position,
                                                                       head_dim, slots, window);
  INK_CHECK_LAUNCH("update_kv");
  return kOk;
}
