// Two 32-bit numbers in one register pair, for the instructions that work on both (each half rounded as
// by fmaf, *, +): the FMA pipes take such an instruction at the rate of one for a single number.
#pragma once

namespace {

using FloatPair = unsigned long long;

__device__ __forceinline__ FloatPair pair_of(float lo, float hi) {
    FloatPair p;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(lo), "f"(hi));
    return p;
}
__device__ __forceinline__ FloatPair pair_of(float x) {
    FloatPair p;
    asm("mov.b64 %0, {%1, %1};" : "=l"(p) : "f"(x));
    return p;
}
__device__ __forceinline__ void unpair(FloatPair p, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p));
}
__device__ __forceinline__ FloatPair fma_pair(FloatPair a, FloatPair b, FloatPair c) {
    FloatPair d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ FloatPair mul_pair(FloatPair a, FloatPair b) {
    FloatPair d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ FloatPair add_pair(FloatPair a, FloatPair b) {
    FloatPair d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// In place, for loops over many sums kept in registers (the 32-bit tiles lose 0.6 % to the form above).
__device__ __forceinline__ void accumulate_pair(FloatPair& acc, FloatPair a, FloatPair b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ void accumulate_pair(FloatPair& acc, FloatPair a) {
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(acc) : "l"(a));
}

}  // namespace
