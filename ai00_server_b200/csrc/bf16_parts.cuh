// f32 numbers as sums of bf16 parts: what the attention kernels of prompt steps (prompt_attn.cuh, latent_prompt.cuh) stage for the tensor core.
#pragma once
#include <cuda_bf16.h>
#include "common.cuh"
#include "linear.cuh"

namespace b200 {

// shared memory only: the general form also waits for the global loads in flight (the next keys)
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(p));
    return p != 0;
}
// 32 lanes x 8 consecutive columns of tensor memory
__device__ __forceinline__ void tc_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// (a, b) -> packed bf16, and what it leaves of them
__device__ __forceinline__ uint32_t pt_take(float& a, float& b) {
    const uint32_t h = pack_bf16x2(make_float2(a, b));
    a -= __uint_as_float(h << 16);
    b -= __uint_as_float(h & 0xFFFF0000u);
    return h;
}

// eight neighbouring numbers, zeros from `left` on (a multiple of four).  WHOLE: `left` is a multiple of eight and the address one of 32 bytes: one access of a whole sector a
// lane (two of 16 bytes, each half of 32 sectors, took 150 us where this takes 130: 16 sequences, contexts of 1024)
template <bool WHOLE>
__device__ __forceinline__ void pt_load8(float (&v)[8], const float* src, const int left) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = 0.f;
    if constexpr (WHOLE) {
        if (left <= 0) return;
        asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                     : "l"(src));
    } else {
#pragma unroll
        for (int i = 0; i < 8; i += 4) {
            const float4 x = i < left ? *reinterpret_cast<const float4*>(src + i) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[i] = x.x; v[i + 1] = x.y; v[i + 2] = x.z; v[i + 3] = x.w;
        }
    }
}

// eight numbers -> the 16 bytes of each of N parts: the first N - 1 rounded to nearest, each takes what those before it left (three parts: all 24 bits, two: 16)
template <int N>
__device__ __forceinline__ void pt_split8(float (&v)[8], uint4 (&part)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) part[i] = make_uint4(pt_take(v[0], v[1]), pt_take(v[2], v[3]), pt_take(v[4], v[5]), pt_take(v[6], v[7]));
}

}  // namespace b200
