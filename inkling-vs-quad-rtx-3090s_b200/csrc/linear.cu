// Dense BF16 projections of up to eight tokens: y = x . W^T, with an optional scalar factor, and the gated pair
// silu(x . G^T) * (x . U^T).
//
// Bound by reading the weights once. One block per SM takes an equal share of the rows, up to eighty at a time. Four warps copy
// them into a ring of stages (256 columns of all rows; cp.async, so that rows lie on a pitch without bank conflicts), a fifth the
// tokens' columns; a consumer warp takes sixteen rows and makes m16n8k16 products (M = weight rows, N = tokens: eight tokens are
// far too few for the tcgen05 tiles). Where the caller vouches for the weights (`settled`: the launch in front does not write them) the ring
// fills before the kernel in front has finished; else the weights, like the tokens, are asked for when it has.
//
// The sum over columns runs from the first to the last, sixteen at a time into one FP32 accumulator: a row and a token have the same bits in any
// company. That is also the order of a plain tensor-core GEMM; on the shapes compared (the tests', torch 2.11) the results were the bits of
// the library calls that stood here, and that matters: a decode step of several layers turns any last-bit difference
// into another rounding of a router logit, hence another routing weight. It costs a chain of K / 16 dependent instructions
// a round (55 clocks each), which the loads hide but for few rows of many columns. (Tiles of eight rows with sums cut between eight
// warps, and between two blocks above 4096 columns: 13.9 us for the 17.3 of 4096 x 8192, 15.9 for 16.3 of 11264 x 4096; but the logits of a six-layer
// step then differ by 2.8 % of their norm.)
//
// us a call, calls on different weights one after the other in a graph, settled weights, one token / seven; the library GEMV that stood here; the
// weights at the copy rate (weights that wait for the kernel in front: 11264 x 4096 17.2 / 17.4, 32768 x 4096 44.5 / 44.8 for 43.0 / 43.7, the others
// within 0.1):  11264 x 4096 16.3 / 16.8, 17.1 / 17.5, 14.1;  4096 x 8192 17.3 / 18.2, 21.5 / 21.7, 10.2;  32768 x 4096 41.0 / 42.6, 45.4 / 45.8, 41.0;
// gated 2 x 8192 x 4096 22.0 / 22.8, 31.5 / 30.2 in four launches, 20.5.
#include "../../include/inkling_b200.h"
#include "common.cuh"
#include "mma_bf16.cuh"
#include "pipe.cuh"

namespace ink {

constexpr int kLinTokens = 8;
constexpr int kLinWeightWarps = 4, kLinConsumers = 5;
constexpr int kLinThreads = (kLinConsumers + kLinWeightWarps + 1) * 32;
constexpr int kLinRows = 16;                       // weight rows of a consumer
constexpr int kLinChunk = 256;                     // columns of a stage
constexpr int kLinPitch = kLinChunk * 2 + 32;      // bytes of a row of a stage: four rows of 32 bytes meet no bank twice
constexpr int kLinMostStages = 12;
constexpr int kLinSmem = 144 * 1024;               // of the ring, at most (a step of six layers: 764 us with 96 KB, 725 so, 729 with 200)
constexpr int kLinMostK = 8192;

struct LinearArgs {
  const uint16_t* x;      // [tokens, k]
  const uint16_t* w;      // [n, k]
  const uint16_t* up;     // gated: [n, k]
  const uint16_t* scale;  // [1] or null
  uint16_t* y;            // [tokens, n]
  int tokens, n, k;
  int groups, stages;     // consumers that have rows; stages of the ring
  int settled;            // the kernel in front does not write the weights
  int32_t* status;        // or null: kFlagWaitTimedOut when a wait gave up
};

struct LinearShared {
  uint64_t full[kLinMostStages], empty[kLinMostStages];
  volatile int failed;
};
// (called when the kernel in front has ended: the limit is for this kernel's own copies and products)
__device__ __forceinline__ bool lin_wait(uint64_t* bar, uint32_t parity, LinearShared* sh, int32_t* status) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (sh->failed) return false;
    if (clock64() - t0 > kWaitLimitCycles) {
      sh->failed = 1;
      if (status) atomicOr(status, kFlagWaitTimedOut);
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ void copy16_async(uint32_t to, const void* from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(from) : "memory");
}
// one arrival of this thread when its copies so far have landed
__device__ __forceinline__ void arrive_when_copied(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// GATED: a consumer's rows 0-7 are gate rows, 8-15 the up rows of the same eight outputs
template <bool GATED>
__global__ void __launch_bounds__(kLinThreads, 1) linear_kernel(const LinearArgs a) {
  constexpr int kOut = GATED ? kLinRows / 2 : kLinRows;   // outputs of a consumer
  extern __shared__ __align__(128) unsigned char s_ring[];   // [stages][groups * 16 + 8 rows][kLinPitch]: weights, then tokens
  __shared__ LinearShared sh;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int stage_rows = a.groups * kLinRows, stage_bytes = (stage_rows + kLinTokens) * kLinPitch;
  const int first = (int)((long long)a.n * blockIdx.x / gridDim.x), end = (int)((long long)a.n * (blockIdx.x + 1) / gridDim.x);
  const int most = a.groups * kOut, rounds = (end - first + most - 1) / most, per_round = rounds > 0 ? (end - first + rounds - 1) / rounds : 0;
  const int chunks = (a.k + kLinChunk - 1) / kLinChunk;
  if (tid == 0) {
    for (int s = 0; s < a.stages; ++s) {
      mbar_init(&sh.full[s], (kLinWeightWarps + 1) * 32);
      mbar_init(&sh.empty[s], (uint32_t)a.groups);
    }
    sh.failed = 0;
    mbar_init_fence();
  }
  __syncthreads();
  if (warp >= kLinConsumers) {
    // =========================================================== copies
    const int producer = warp - kLinConsumers;
    const bool weights = producer < kLinWeightWarps;
    if (!weights || !a.settled) pdl_wait();   // x is there now, and any weights
    if (!weights) pdl_trigger();
    const uint32_t ring = smem_u32(s_ring);
    int stage = 0;
    uint32_t lap = 0;
    bool ok = true;
    for (int round = 0; ok && round < rounds; ++round) {
      const int row0 = first + round * per_round, outputs = min(per_round, end - row0);
      for (int c = 0; c < chunks; ++c) {
        if (lap > 0) {
          if (lap == 1 && stage == 0) pdl_wait();   // (the products start when the kernel in front has ended)
          ok = __all_sync(0xffffffffu, lin_wait(&sh.empty[stage], (lap - 1) & 1u, &sh, a.status));
        }
        if (!ok) break;
        const int k0 = c * kLinChunk + lane * 8;
        const uint32_t to = ring + (uint32_t)(stage * stage_bytes) + (uint32_t)lane * 16;
        if (k0 < a.k) {
          if (weights) {
#pragma unroll 4
            for (int r = producer; r < (GATED ? 2 * outputs : outputs); r += kLinWeightWarps) {
              const int i = GATED ? r >> 1 : r, slot = GATED ? (i >> 3) * kLinRows + (r & 1) * 8 + (i & 7) : r;
              copy16_async(to + (uint32_t)(slot * kLinPitch), (GATED && (r & 1) ? a.up : a.w) + (size_t)(row0 + i) * a.k + k0);
            }
          } else {
            for (int j = 0; j < a.tokens; ++j) copy16_async(to + (uint32_t)((stage_rows + j) * kLinPitch), a.x + (size_t)j * a.k + k0);
          }
        }
        arrive_when_copied(&sh.full[stage]);
        if (++stage == a.stages) {
          stage = 0;
          ++lap;
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp < a.groups) {
    // =========================================================== products
    const int g = lane >> 2, t = lane & 3;
    const unsigned char* rows = s_ring + (warp * kLinRows + g) * kLinPitch + t * 8;        // (rows beyond the share hold anything: they
    const unsigned char* tokens = s_ring + (stage_rows + g) * kLinPitch + t * 8;           //  and tokens beyond the last are not written)
    pdl_wait();   // (the tokens; and y may still be read by the kernels in front)
    int stage = 0;
    uint32_t lap = 0;
    bool ok = true;
    for (int round = 0; round < rounds; ++round) {
      float d[4] = {0.f, 0.f, 0.f, 0.f};
      for (int c = 0; ok && c < chunks; ++c) {
        ok = __all_sync(0xffffffffu, lin_wait(&sh.full[stage], lap & 1u, &sh, a.status));
        if (!ok) break;
        const unsigned char *w = rows + stage * stage_bytes, *x = tokens + stage * stage_bytes;
        // (a lane's four columns of a step are neighbours, on both sides: the sum over sixteen does not depend on who holds which)
        struct Operands { uint2 w0, w1, x; };
        auto fetch = [&](int i) -> Operands {
          return {*reinterpret_cast<const uint2*>(w + i * 32), *reinterpret_cast<const uint2*>(w + 8 * kLinPitch + i * 32), *reinterpret_cast<const uint2*>(x + i * 32)};
        };
        auto product = [&](const Operands& o) { mma_bf16(d, o.w0.x, o.w1.x, o.w0.y, o.w1.y, o.x.x, o.x.y); };
        const int steps = min(kLinChunk, a.k - c * kLinChunk) / 16;
        if (steps == kLinChunk / 16) {
          constexpr int kAhead = 8;   // the products are a chain, their operands need not be
          Operands o[kAhead];
#pragma unroll
          for (int i = 0; i < kAhead; ++i) o[i] = fetch(i);
#pragma unroll
          for (int i = 0; i < kLinChunk / 16; ++i) {
            product(o[i % kAhead]);
            if (i + kAhead < kLinChunk / 16) o[i % kAhead] = fetch(i + kAhead);
          }
        } else {
          for (int i = 0; i < steps; ++i) product(fetch(i));
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.empty[stage]);
        if (++stage == a.stages) {
          stage = 0;
          ++lap;
        }
      }
      if (!ok) d[0] = d[1] = d[2] = d[3] = __int_as_float(0x7fffffff);   // (a wait that gave up shows in the results)
      const int row0 = first + round * per_round, outputs = min(per_round, end - row0);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int out = warp * kOut + g + (GATED ? 0 : j >> 1) * 8, token = 2 * t + (j & 1);
        if ((GATED && j >= 2) || out >= outputs || token >= a.tokens) continue;
        float v = round_bf16(d[j]);
        if (GATED) v = round_bf16(round_bf16(v / (1.f + expf(-v))) * round_bf16(d[(j & 1) + 2]));   // as the BF16 tensor operations round
        if (a.scale) v = v * bf16_to_f32(a.scale[0]);
        a.y[(size_t)token * a.n + row0 + out] = (uint16_t)f32_to_bf16_bits(v);
      }
    }
  }
  __syncwarp();
  pdl_wait();   // whoever waits for this kernel may rely on the ones before it too
}

template <bool GATED>
static int launch_linear(LinearArgs a, cudaStream_t stream) {
  constexpr int kMaxDevices = 64;
  static int sms_of[kMaxDevices] = {};   // 0: this device is not configured yet
  int device = 0;
  cudaGetDevice(&device);
  INK_REQUIRE(device >= 0 && device < kMaxDevices, kLaunchFailed, "linear: device ordinal %d", device);
  if (sms_of[device] == 0) {
    const cudaError_t e = cudaFuncSetAttribute(linear_kernel<GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, kLinSmem);
    INK_REQUIRE(e == cudaSuccess, kLaunchFailed, "linear: %d bytes of shared memory refused: %s", kLinSmem, cudaGetErrorString(e));
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    sms_of[device] = sms > 0 ? sms : 148;
  }
  const int blocks = a.n < sms_of[device] ? a.n : sms_of[device], out = GATED ? kLinRows / 2 : kLinRows;
  const int share = (a.n + blocks - 1) / blocks, rounds = (share + kLinConsumers * out - 1) / (kLinConsumers * out);
  a.groups = ((share + rounds - 1) / rounds + out - 1) / out;
  const int stage = (a.groups * kLinRows + kLinTokens) * kLinPitch, chunks = (a.k + kLinChunk - 1) / kLinChunk * rounds;
  a.stages = kLinSmem / stage;
  if (a.stages > kLinMostStages) a.stages = kLinMostStages;
  if (a.stages > chunks) a.stages = chunks;
  static_assert(kLinSmem / ((kLinConsumers * kLinRows + kLinTokens) * kLinPitch) >= 2, "the ring holds two stages");
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3((unsigned)blocks);
  config.blockDim = dim3(kLinThreads);
  config.dynamicSmemBytes = (size_t)a.stages * stage;
  config.stream = stream;
  cudaLaunchAttribute attribute;
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  config.attrs = &attribute;
  config.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&config, linear_kernel<GATED>, a);
  INK_REQUIRE(e == cudaSuccess, kLaunchFailed, "linear: launch failed: %s", cudaGetErrorString(e));
  return kOk;
}

}  // namespace ink

using namespace ink;

extern "C" int ink_linear_settled(const void* x, const void* weight, const void* up, const void* scale, void* y, int tokens, int n, int k,
                                  int settled, int32_t* status, ink_stream_t stream) {
  INK_REQUIRE(x && weight && y, kBadArgument, "linear: null pointer argument");
  INK_REQUIRE(tokens >= 0 && tokens <= kLinTokens && n > 0 && n <= (1 << 24) && k > 0 && k % 32 == 0 && k <= kLinMostK, kUnsupportedShape,
              "linear: tokens=%d n=%d k=%d unsupported (up to %d tokens, k a multiple of 32 up to %d)", tokens, n, k, kLinTokens, kLinMostK);
  INK_REQUIRE(aligned16(x) && aligned16(weight) && aligned16(up), kMisaligned, "linear: x and weights must be 16-byte aligned");
  if (tokens == 0) return kOk;
  const LinearArgs a{(const uint16_t*)x, (const uint16_t*)weight, (const uint16_t*)up, (const uint16_t*)scale, (uint16_t*)y, tokens, n, k, 0, 0, settled, status};
  return up ? launch_linear<true>(a, (cudaStream_t)stream) : launch_linear<false>(a, (cudaStream_t)stream);
}

extern "C" int ink_linear(const void* x, const void* weight, const void* up, const void* scale, void* y, int tokens, int n, int k,
                          ink_stream_t stream) {
  return ink_linear_settled(x, weight, up, scale, y, tokens, n, k, 0, nullptr, stream);
}
