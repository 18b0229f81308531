// Packed pairs of f32: two IEEE operations an instruction (sm_100's fma.rn.f32x2 and its kin), each rounded as the single one would be.  The multiply-add
// rate is that of single instructions (36 and 37 T multiply-adds a second); what they save is issue slots beside loads and exchanges.
#pragma once
#include <stdint.h>

namespace b200 {

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ void fma2(f32x2& acc, f32x2 a, f32x2 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }      // acc += a b
__device__ __forceinline__ f32x2 fmadd2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ void mul2(f32x2& acc, f32x2 a) { asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(acc) : "l"(a)); }
__device__ __forceinline__ f32x2 prod2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

}  // namespace b200
