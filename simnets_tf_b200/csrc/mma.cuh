// Warp-sized TF32 tensor-core products (m16n8k8) for contractions that are slivers of another kernel's tile.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace simnets {

// d[16 x 8] += a[16 x 8] b[8 x 8].  lane = 4 q + t: a = (q, t), (q + 8, t), (q, t + 4), (q + 8, t + 4); b = (t, q), (t + 4, q);
// d = (q, 2t), (q, 2t + 1), (q + 8, 2t), (q + 8, 2t + 1).  What is added to d is truncated: keep sums over many products elsewhere.
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// v = hi + lo exactly, hi with the bits a TF32 operand keeps
__device__ __forceinline__ float2 split_tf32(float v) {
    const float hi = __uint_as_float(__float_as_uint(v) & 0xffffe000u);
    return make_float2(hi, v - hi);
}

}  // namespace simnets
