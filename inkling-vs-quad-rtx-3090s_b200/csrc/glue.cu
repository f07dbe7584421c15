// What stands between the projections, the attention and the expert block of a decoder layer at decode: norms, short
// convolutions, residuals. All of it is latency: a few rows, read and written once.
#include "../../include/inkling_b200.h"
#include "common.cuh"
#include "mma_bf16.cuh"

namespace ink {

constexpr int kNormThreads = 256;
constexpr int kNormMaxPerThread = 8;  // 8-element groups per thread: hidden <= 256 * 8 * 8

// Residual add + RMS norm between two MoE blocks: one block per token. Without ADD the norm alone, `residual` is left as it is
// (4 096 elements, seven tokens: 1.7 us for a copy of the rows and 3.9 with zeros added to them; 3.9 so, most of it beside the kernel in front).
template <bool ADD>
__global__ void __launch_bounds__(kNormThreads) add_rmsnorm_kernel(const float* __restrict__ partial,
                                                                    uint16_t* __restrict__ residual,
                                                                    const uint16_t* __restrict__ weight, float eps,
                                                                    uint16_t* __restrict__ normed, int hidden) {
  __shared__ float s_red[kNormThreads / 32];
  pdl_wait();
  pdl_trigger();
  const int token = blockIdx.x, tid = threadIdx.x;
  const float* p = ADD ? partial + (size_t)token * hidden : nullptr;
  uint16_t* r = residual + (size_t)token * hidden;
  uint16_t* y = normed + (size_t)token * hidden;
  const int groups = hidden / 8;
  float h[kNormMaxPerThread][8];
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < kNormMaxPerThread; ++i) {
    const int gidx = i * kNormThreads + tid;
    if (gidx < groups) {
      const float4 a = ADD ? __ldcg(reinterpret_cast<const float4*>(p + gidx * 8)) : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 b = ADD ? __ldcg(reinterpret_cast<const float4*>(p + gidx * 8 + 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
      const uint4 q = __ldcg(reinterpret_cast<const uint4*>(r + gidx * 8));
      const float add[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
      const uint32_t res[4] = {q.x, q.y, q.z, q.w};
      uint32_t packed[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float lo = round_bf16(bf16lo(res[j]) + round_bf16(add[2 * j]));
        const float hi = round_bf16(bf16hi(res[j]) + round_bf16(add[2 * j + 1]));
        h[i][2 * j] = lo;
        h[i][2 * j + 1] = hi;
        sum = fmaf(lo, lo, sum);
        sum = fmaf(hi, hi, sum);
        packed[j] = f32_to_bf16_bits(lo) | (f32_to_bf16_bits(hi) << 16);
      }
      if (ADD) *reinterpret_cast<uint4*>(r + gidx * 8) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    }
  }
  sum = warp_sum(sum);
  if ((tid & 31) == 0) s_red[tid >> 5] = sum;
  __syncthreads();
  float total = 0.f;
#pragma unroll
  for (int w = 0; w < kNormThreads / 32; ++w) total += s_red[w];
  const float scale = rsqrtf(total / (float)hidden + eps);
#pragma unroll
  for (int i = 0; i < kNormMaxPerThread; ++i) {
    const int gidx = i * kNormThreads + tid;
    if (gidx < groups) {
      const uint4 wq = __ldcg(reinterpret_cast<const uint4*>(weight + gidx * 8));
      const uint32_t wv[4] = {wq.x, wq.y, wq.z, wq.w};
      uint32_t packed[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float lo = round_bf16(h[i][2 * j] * scale) * bf16lo(wv[j]);
        const float hi = round_bf16(h[i][2 * j + 1] * scale) * bf16hi(wv[j]);
        packed[j] = f32_to_bf16_bits(lo) | (f32_to_bf16_bits(hi) << 16);
      }
      *reinterpret_cast<uint4*>(y + gidx * 8) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    }
  }
}

// One channel of the short convolution. Fetched apart from its use: a kernel that stores one channel's history before it asks for the
// next one's waits for each in turn. WIDE: four taps, taps and history 16-byte aligned.
template <int TAPS, bool WIDE>
struct ConvChannel {
  float past[TAPS], tap[TAPS];
  __device__ __forceinline__ void fetch(const float* taps, const float* history) {
    if constexpr (WIDE) {
      const float4 h = __ldcg(reinterpret_cast<const float4*>(history)), w = __ldcg(reinterpret_cast<const float4*>(taps));
      past[0] = h.x; past[1] = h.y; past[2] = h.z; past[3] = h.w;
      tap[0] = w.x; tap[1] = w.y; tap[2] = w.z; tap[3] = w.w;
    } else {
#pragma unroll
      for (int j = 0; j < TAPS; ++j) {
        past[j] = __ldcg(history + j);
        tap[j] = __ldcg(taps + j);
      }
    }
  }
  // The new output, before any residual; the history moves on by one. Separate multiplies and adds in tap order, as the
  // reference kernel computes them (no fused multiply-add).
  __device__ __forceinline__ float step(float current, float* history) const {
    float total = 0.f;
#pragma unroll
    for (int j = 0; j + 1 < TAPS; ++j) total = __fadd_rn(total, __fmul_rn(past[j + 1], tap[j]));
    total = __fadd_rn(total, __fmul_rn(current, tap[TAPS - 1]));
    if constexpr (WIDE) {
      *reinterpret_cast<float4*>(history) = make_float4(past[1], past[2], past[3], current);
    } else {
#pragma unroll
      for (int j = 0; j + 1 < TAPS; ++j) history[j] = past[j + 1];
      history[TAPS - 1] = current;
    }
    return round_bf16(__fadd_rn(total, current));
  }
};

// Short convolution of one new token per sequence with its cached FP32 history, the skip
// connection and the decoder residual: one thread per channel. XF32 = 1: x is the block's
// FP32 output, cast to BF16 first (what the expert runtime returns to the layer).
template <int TAPS, bool XF32, bool WIDE>
__global__ void __launch_bounds__(256) short_conv_kernel(const void* __restrict__ x_raw, const float* __restrict__ taps,
                                                          float* __restrict__ history, const uint16_t* __restrict__ residual,
                                                          uint16_t* __restrict__ y, int hidden) {
  pdl_wait();
  pdl_trigger();
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= hidden) return;
  const size_t at = (size_t)blockIdx.y * hidden + d;
  float current;
  if (XF32) current = round_bf16(__ldcg(reinterpret_cast<const float*>(x_raw) + at));
  else current = bf16_to_f32(__ldcg(reinterpret_cast<const uint16_t*>(x_raw) + at));
  ConvChannel<TAPS, WIDE> conv;
  conv.fetch(taps + (size_t)d * TAPS, history + at * TAPS);
  float out = conv.step(current, history + at * TAPS);
  if (residual) out = round_bf16(__fadd_rn(out, bf16_to_f32(__ldcg(residual + at))));
  y[at] = (uint16_t)f32_to_bf16_bits(out);
}

// The same with the norm of the sum that follows it (attn_sconv, residual, post-attention norm), BF16 in. Eight blocks, a
// cluster, per token: block w takes the channels that warp w of add_rmsnorm_kernel takes and its warp 0 sums their squares as that warp does,
// so the norm comes out in the same bits. (A row's history and taps, 128 KB at 4 096 channels, are too much for one SM.)
constexpr int kConvNormBlocks = kNormThreads / 32, kConvNormThreads = 128;
template <int TAPS>
__global__ void __launch_bounds__(kConvNormThreads) conv_norm_kernel(const uint16_t* __restrict__ x, const float* __restrict__ taps,
                                                                      float* __restrict__ history, const uint16_t* __restrict__ residual,
                                                                      const uint16_t* __restrict__ weight, float eps, uint16_t* __restrict__ y,
                                                                      uint16_t* __restrict__ normed, int hidden) {
  __shared__ float s_h[kNormMaxPerThread * 256];   // this block's sums: 256 channels of every 2 048
  __shared__ float s_sum;
  pdl_wait();
  pdl_trigger();
  const int rank = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
  const size_t row = (size_t)blockIdx.y * hidden;
  auto channel_of = [&](int i) -> int { return i / 256 * (kNormThreads * 8) + rank * 256 + i % 256; };
  constexpr int kAhead = 4;   // channels of a thread at a time: all of them up to 4 096 in all
#pragma unroll 1
  for (int i0 = tid; channel_of(i0) < hidden; i0 += kAhead * kConvNormThreads) {
    ConvChannel<TAPS, TAPS == 4> conv[kAhead];
    float in[kAhead], skip[kAhead];
#pragma unroll
    for (int n = 0; n < kAhead; ++n) {
      const int d = channel_of(i0 + n * kConvNormThreads);
      if (d >= hidden) continue;
      conv[n].fetch(taps + (size_t)d * TAPS, history + (row + d) * TAPS);
      in[n] = bf16_to_f32(__ldcg(x + row + d));
      skip[n] = bf16_to_f32(__ldcg(residual + row + d));
    }
#pragma unroll
    for (int n = 0; n < kAhead; ++n) {
      const int i = i0 + n * kConvNormThreads, d = channel_of(i);
      if (d >= hidden) continue;
      const float out = round_bf16(__fadd_rn(conv[n].step(in[n], history + (row + d) * TAPS), skip[n]));
      y[row + d] = (uint16_t)f32_to_bf16_bits(out);
      s_h[i] = round_bf16(out + 0.f);
    }
  }
  __syncthreads();
  if (tid < 32) {
    float sum = 0.f;
    for (int i = lane * 8; channel_of(i) < hidden; i += 256)
#pragma unroll
      for (int j = 0; j < 8; ++j) sum = fmaf(s_h[i + j], s_h[i + j], sum);
    sum = warp_sum(sum);
    if (lane == 0) s_sum = sum;
  }
  cluster_sync();
  float part[kConvNormBlocks], total = 0.f;
#pragma unroll
  for (int w = 0; w < kConvNormBlocks; ++w) part[w] = ld_cluster_float(&s_sum, w);
#pragma unroll
  for (int w = 0; w < kConvNormBlocks; ++w) total += part[w];
  const float scale = rsqrtf(total / (float)hidden + eps);
  for (int i = tid; channel_of(i) < hidden; i += kConvNormThreads) {
    const int d = channel_of(i);
    normed[row + d] = (uint16_t)f32_to_bf16_bits(round_bf16(s_h[i] * scale) * bf16_to_f32(__ldcg(weight + d)));
  }
  cluster_sync();   // (a block's sum stays until all have read it)
}

// Between the fused projection and the attention: norm of the query heads, short convolution and norm of the keys, short
// convolution of the values, relative states; one warp per head, eight elements a lane (what add_rmsnorm_kernel's first warp does
// with a row of up to 256). In eight launches with the copies between them this took 21 us for seven sequences of 64 + 2 x 8 heads of 128, 4.5 so
// (every lane asks for all it needs before it stores anything: one after the other, as aliasing pointers make the compiler keep
// them, 10 us).
struct HeadsArgs {
  const uint16_t* qkvr;   // [batch, (h + 2 hk) c + h d_rel]
  const uint16_t *q_weight, *k_weight;
  const float *k_taps, *v_taps;
  float *k_history, *v_history;
  uint16_t *q, *k, *v, *r;
  int batch, heads, kv_heads, head_dim, d_rel;
  float eps;
};
template <int TAPS>
__global__ void __launch_bounds__(128) heads_kernel(const HeadsArgs a) {
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31, c = a.head_dim, width = (a.heads + 2 * a.kv_heads) * c + a.heads * a.d_rel;
  const int vectors = a.heads + 2 * a.kv_heads + 1;   // of a token; the last is its relative states
  const int at = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (at >= a.batch * vectors) return;
  const int b = at / vectors, n = at % vectors;
  const uint16_t* from = a.qkvr + (size_t)b * width + (size_t)n * c;
  if (n == vectors - 1) {
    const int pieces = a.heads * a.d_rel / 8;
    uint4* to = reinterpret_cast<uint4*>(a.r) + (size_t)b * pieces;
    for (int i0 = lane; i0 < pieces; i0 += 128) {   // (all of a round asked for before any is stored)
      uint4 v[4];
#pragma unroll
      for (int n = 0; n < 4; ++n) v[n] = i0 + 32 * n < pieces ? __ldcg(reinterpret_cast<const uint4*>(from) + i0 + 32 * n) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int n = 0; n < 4; ++n)
        if (i0 + 32 * n < pieces) to[i0 + 32 * n] = v[n];
    }
    return;
  }
  const bool live = lane * 8 < c;
  float h[8];
  {
    const uint4 raw = live ? __ldcg(reinterpret_cast<const uint4*>(from) + lane) : make_uint4(0, 0, 0, 0);
    const uint32_t in[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      h[2 * j] = bf16lo(in[j]);
      h[2 * j + 1] = bf16hi(in[j]);
    }
  }
  const uint16_t* weight = a.q_weight;
  uint16_t* to = a.q + ((size_t)b * a.heads + n) * c;
  if (n >= a.heads) {
    const bool value = n >= a.heads + a.kv_heads;
    const int head = n - a.heads - (value ? a.kv_heads : 0), d = head * c + lane * 8;
    const float* taps = (value ? a.v_taps : a.k_taps) + (size_t)d * TAPS;
    float* history = (value ? a.v_history : a.k_history) + ((size_t)b * a.kv_heads * c + d) * TAPS;
    if (live) {
      ConvChannel<TAPS, TAPS == 4> conv[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) conv[j].fetch(taps + j * TAPS, history + j * TAPS);
#pragma unroll
      for (int j = 0; j < 8; ++j) h[j] = conv[j].step(h[j], history + j * TAPS);
    }
    to = (value ? a.v : a.k) + ((size_t)b * a.kv_heads + head) * c;
    weight = value ? nullptr : a.k_weight;
  }
  if (weight) {
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      h[j] = round_bf16(h[j] + 0.f);
      sum = fmaf(h[j], h[j], sum);
    }
    sum = warp_sum(sum);
    const float scale = rsqrtf(sum / (float)c + a.eps);
    const uint4 raw = live ? __ldcg(reinterpret_cast<const uint4*>(weight) + lane) : make_uint4(0, 0, 0, 0);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      h[2 * j] = round_bf16(h[2 * j] * scale) * bf16lo(w[j]);
      h[2 * j + 1] = round_bf16(h[2 * j + 1] * scale) * bf16hi(w[j]);
    }
  }
  if (live) {
    uint32_t out[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) out[j] = f32_to_bf16_bits(h[2 * j]) | (f32_to_bf16_bits(h[2 * j + 1]) << 16);
    *(reinterpret_cast<uint4*>(to) + lane) = make_uint4(out[0], out[1], out[2], out[3]);
  }
}

// A launch that may start while the kernel in front runs (see pdl_wait). What that one writes is read through L2, never by loads
// that are meant for memory nobody writes while a kernel is there.
template <typename... Params, typename... Args>
static cudaError_t launch_after(void (*kernel)(Params...), dim3 grid, int threads, int cluster, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = dim3((unsigned)threads);
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[0].val.programmaticStreamSerializationAllowed = 1;
  attributes[1].id = cudaLaunchAttributeClusterDimension;
  attributes[1].val.clusterDim.x = (unsigned)cluster;
  attributes[1].val.clusterDim.y = attributes[1].val.clusterDim.z = 1;
  config.attrs = attributes;
  config.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}

}  // namespace ink

using namespace ink;

extern "C" int ink_short_conv(const void* x, int x_is_fp32, const float* taps, float* history, const void* residual,
                              void* y, int batch, int hidden, int kernel_size, ink_stream_t stream) {
  INK_REQUIRE(x && taps && history && y, kBadArgument, "short_conv: null pointer argument");
  INK_REQUIRE(batch >= 0 && hidden > 0, kBadArgument, "short_conv: batch=%d hidden=%d", batch, hidden);
  INK_REQUIRE(kernel_size >= 2 && kernel_size <= 4, kUnsupportedShape, "short_conv: kernel_size=%d (2..4 are built)",
              kernel_size);
  if (batch == 0) return kOk;
  const dim3 grid((unsigned)((hidden + 255) / 256), (unsigned)batch);
  cudaStream_t s = (cudaStream_t)stream;
  const uint16_t* r = (const uint16_t*)residual;
  uint16_t* out = (uint16_t*)y;
  cudaError_t e = cudaSuccess;
  const bool wide = kernel_size == 4 && aligned16(taps) && aligned16(history);
#define INK_SCONV_CASE(T, W)                                                                                                                   \
  if (kernel_size == T && wide == W)                                                                                                           \
    e = launch_after(x_is_fp32 ? short_conv_kernel<T, true, W> : short_conv_kernel<T, false, W>, grid, 256, 1, s, x, taps, history, r, out, hidden);
  INK_SCONV_CASE(2, false)
  INK_SCONV_CASE(3, false)
  INK_SCONV_CASE(4, false)
  INK_SCONV_CASE(4, true)
#undef INK_SCONV_CASE
  INK_REQUIRE(e == cudaSuccess, kLaunchFailed, "short_conv: launch failed: %s", cudaGetErrorString(e));
  return kOk;
}

extern "C" int ink_add_rmsnorm(const float* partial, void* residual, const void* weight, float eps, void* normed,
                               int tokens, int hidden, ink_stream_t stream) {
  INK_REQUIRE(partial && residual && weight && normed, kBadArgument, "add_rmsnorm: null pointer argument");
  INK_REQUIRE(tokens >= 0 && hidden > 0 && hidden % 8 == 0 && hidden <= kNormThreads * kNormMaxPerThread * 8,
              kUnsupportedShape, "add_rmsnorm: tokens=%d hidden=%d unsupported", tokens, hidden);
  INK_REQUIRE(aligned16(partial) && aligned16(residual) && aligned16(weight) && aligned16(normed), kMisaligned,
              "add_rmsnorm: buffers must be 16-byte aligned");
  if (tokens == 0) return kOk;
  INK_PREFER_MAX_SMEM(add_rmsnorm_kernel<true>);
  const cudaError_t e = launch_after(add_rmsnorm_kernel<true>, dim3(tokens), kNormThreads, 1, (cudaStream_t)stream, partial, (uint16_t*)residual,
                                     (const uint16_t*)weight, eps, (uint16_t*)normed, hidden);
  INK_REQUIRE(e == cudaSuccess, kLaunchFailed, "add_rmsnorm: launch failed: %s", cudaGetErrorString(e));
  return kOk;
}

extern "C" int ink_rmsnorm(const void* x, const void* weight, float eps, void* normed, int tokens, int hidden, ink_stream_t stream) {
  INK_REQUIRE(x && weight && normed, kBadArgument, "rmsnorm: null pointer argument");
  INK_REQUIRE(tokens >= 0 && hidden > 0 && hidden % 8 == 0 && hidden <= kNormThreads * kNormMaxPerThread * 8,
              kUnsupportedShape, "rmsnorm: tokens=%d hidden=%d unsupported", tokens, hidden);
  INK_REQUIRE(aligned16(x) && aligned16(weight) && aligned16(normed), kMisaligned, "rmsnorm: buffers must be 16-byte aligned");
  if (tokens == 0) return kOk;
  const cudaError_t e = launch_after(add_rmsnorm_kernel<false>, dim3(tokens), kNormThreads, 1, (cudaStream_t)stream, nullptr, (uint16_t*)const_cast<void*>(x),
                                     (const uint16_t*)weight, eps, (uint16_t*)normed, hidden);
  INK_REQUIRE(e == cudaSuccess, kLaunchFailed, "rmsnorm: launch failed: %s", cudaGetErrorString(e));
  return kOk;
}

extern "C" int ink_short_conv_norm(const void* x, const float* taps, float* history, const void* residual, const void* weight, float eps, void* y,
                                   void* normed, int batch, int hidden, int kernel_size, ink_stream_t stream) {
  INK_REQUIRE(x && taps && history && residual && weight && y && normed, kBadArgument, "short_conv_norm: null pointer argument");
  INK_REQUIRE(batch >= 0 && batch <= 65535 && hidden > 0 && hidden % 8 == 0 && hidden <= kNormThreads * kNormMaxPerThread * 8, kUnsupportedShape,
              "short_conv_norm: batch=%d hidden=%d unsupported", batch, hidden);
  INK_REQUIRE(kernel_size >= 2 && kernel_size <= 4, kUnsupportedShape, "short_conv_norm: kernel_size=%d (2..4 are built)", kernel_size);
  INK_REQUIRE(aligned16(taps) && aligned16(history), kMisaligned, "short_conv_norm: taps and history must be 16-byte aligned");
  if (batch == 0) return kOk;
  const auto kernel = kernel_size == 4 ? conv_norm_kernel<4> : kernel_size == 3 ? conv_norm_kernel<3> : conv_norm_kernel<2>;
  const cudaError_t e = launch_after(kernel, dim3(kConvNormBlocks, (unsigned)batch), kConvNormThreads, kConvNormBlocks, (cudaStream_t)stream, (const uint16_t*)x, taps,
                                     history, (const uint16_t*)residual, (const uint16_t*)weight, eps, (uint16_t*)y, (uint16_t*)normed, hidden);
  INK_REQUIRE(e == cudaSuccess, kLaunchFailed, "short_conv_norm: launch failed: %s", cudaGetErrorString(e));
  return kOk;
}

extern "C" int ink_attention_heads(const void* qkvr, const void* q_weight, const void* k_weight, const float* k_taps, const float* v_taps, float* k_history,
                                   float* v_history, float eps, void* q, void* k, void* v, void* r, int batch, int heads, int kv_heads, int head_dim,
                                   int d_rel, int kernel_size, ink_stream_t stream) {
  INK_REQUIRE(qkvr && q_weight && k_weight && k_taps && v_taps && k_history && v_history && q && k && v && r, kBadArgument,
              "attention_heads: null pointer argument");
  INK_REQUIRE(batch >= 0 && heads > 0 && kv_heads > 0 && head_dim > 0 && head_dim % 8 == 0 && head_dim <= 256 && d_rel >= 0 && (heads * d_rel) % 8 == 0,
              kUnsupportedShape, "attention_heads: batch=%d heads=%d kv_heads=%d head_dim=%d d_rel=%d unsupported", batch, heads, kv_heads, head_dim, d_rel);
  INK_REQUIRE(kernel_size >= 2 && kernel_size <= 4, kUnsupportedShape, "attention_heads: kernel_size=%d (2..4 are built)", kernel_size);
  INK_REQUIRE(aligned16(qkvr) && aligned16(q_weight) && aligned16(k_weight) && aligned16(k_taps) && aligned16(v_taps) && aligned16(k_history) &&
                  aligned16(v_history) && aligned16(q) && aligned16(k) && aligned16(v) && aligned16(r),
              kMisaligned, "attention_heads: buffers must be 16-byte aligned");
  if (batch == 0) return kOk;
  const long long vectors = (long long)batch * (heads + 2 * kv_heads + 1);
  INK_REQUIRE(vectors <= 0x7fffffff, kUnsupportedShape, "attention_heads: %lld heads in one call", vectors);
  const HeadsArgs a{(const uint16_t*)qkvr, (const uint16_t*)q_weight, (const uint16_t*)k_weight, k_taps, v_taps, k_history, v_history,
                    (uint16_t*)q, (uint16_t*)k, (uint16_t*)v, (uint16_t*)r, batch, heads, kv_heads, head_dim, d_rel, eps};
  const auto kernel = kernel_size == 4 ? heads_kernel<4> : kernel_size == 3 ? heads_kernel<3> : heads_kernel<2>;
  const cudaError_t e = launch_after(kernel, dim3((unsigned)((vectors + 3) / 4)), 128, 1, (cudaStream_t)stream, a);
  INK_REQUIRE(e == cudaSuccess, kLaunchFailed, "attention_heads: launch failed: %s", cudaGetErrorString(e));
  return kOk;
}
