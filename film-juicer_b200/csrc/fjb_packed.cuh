// fjb_packed.cuh -- two FP32 values in one 64-bit register. Every operation rounds each half
// as the scalar instruction does; one issue slot serves both.
#pragma once

#include <cuda_runtime.h>

namespace fjb {

struct Pair {
    unsigned long long v;
};
__device__ __forceinline__ Pair pack(float a, float b) {
    Pair r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack(Pair p) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p.v));
    return r;
}
__device__ __forceinline__ Pair fma2(Pair a, Pair b, Pair c) {
    Pair r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ Pair mul2(Pair a, Pair b) {
    Pair r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ Pair add2(Pair a, Pair b) {
    Pair r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
// a - b (b's product with -1 is exact)
__device__ __forceinline__ Pair sub2(Pair a, Pair b) { return fma2(b, pack(-1.0f, -1.0f), a); }

} // namespace fjb
