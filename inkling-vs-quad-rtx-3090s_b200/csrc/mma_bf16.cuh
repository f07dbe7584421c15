// Warp-level BF16 matrix instructions, thread-block clusters and programmatic dependent launch: what the kernels of the layer
// around the experts share.
#pragma once
#include "common.cuh"

namespace ink {

// D[16x8] += A[16x16] . B[16x8], BF16 in, FP32 out. Lane (g = lane / 4, t = lane % 4) holds of A: a0 = row g,
// columns 2t, 2t+1; a1 = row g + 8, the same columns; a2, a3 = columns 2t+8, 2t+9 of these rows; of B: b0 = rows
// 2t, 2t+1, b1 = rows 2t+8, 2t+9 of column g; of D: d0, d1 = row g, columns 2t, 2t+1; d2, d3 = row g + 8.
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the float(s) at this block's address `p` in the shared memory of block `rank` of the cluster
__device__ __forceinline__ float ld_cluster_float(const float* p, int rank) {
  float v;
  asm volatile("{\n .reg .u32 at;\n mapa.shared::cluster.u32 at, %1, %2;\n ld.shared::cluster.f32 %0, [at];\n}\n"
               : "=f"(v)
               : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank)
               : "memory");
  return v;
}
__device__ __forceinline__ float2 ld_cluster_float2(const float* p, int rank) {
  float2 v;
  asm volatile("{\n .reg .u32 at;\n mapa.shared::cluster.u32 at, %2, %3;\n ld.shared::cluster.v2.f32 {%0, %1}, [at];\n}\n"
               : "=f"(v.x), "=f"(v.y)
               : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank)
               : "memory");
  return v;
}

// Programmatic dependent launch. A kernel launched as a dependent starts when the one in front has let it (every block has
// triggered or ended); what that one wrote is there after pdl_wait, which also means that it has ended. Every block waits
// before it ends, so whoever waits for a kernel may rely on all the kernels before it too. Kernels trigger after their own wait (the
// grouped projections before it: nothing but their own staging and sums follows them): a kernel that has started may rely, without
// waiting, on all that was written before the kernel in front of it.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

}  // namespace ink
