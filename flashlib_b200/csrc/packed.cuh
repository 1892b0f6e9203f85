// Packed fp32 pairs (add / fma on two floats of a 64-bit register): half the issue slots of the scalar forms.
#pragma once
#include "common.cuh"

namespace fl {

__device__ __forceinline__ unsigned long long pk2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpk2(unsigned long long v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// a * a + s
__device__ __forceinline__ unsigned long long sqadd2(unsigned long long a, unsigned long long s) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %1, %2;" : "=l"(r) : "l"(a), "l"(s));
    return r;
}
__device__ __forceinline__ float fold2(unsigned long long a) {
    float lo, hi;
    unpk2(a, lo, hi);
    return lo + hi;
}

}  // namespace fl
