// f32x2.cuh -- paired FP32 arithmetic of the pair sums.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace gsph {

// Paired FP32 (PTX ISA 8.6, sm_100+): one add/sub/mul/fma.rn.f32x2 instruction performs the same
// IEEE single-precision operation on two lanes of a 64-bit register pair, so two i-particles advance
// per issued instruction with bit-identical results to the scalar form.
__device__ __forceinline__ uint64_t u64_of(float2 v) { return *reinterpret_cast<uint64_t*>(&v); }
__device__ __forceinline__ float2 f2_of(uint64_t v) { return *reinterpret_cast<float2*>(&v); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(u64_of(a)), "l"(u64_of(b)), "l"(u64_of(c)));
    return f2_of(d);
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    uint64_t d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(u64_of(a)), "l"(u64_of(b)));
    return f2_of(d);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(u64_of(a)), "l"(u64_of(b)));
    return f2_of(d);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(u64_of(a)), "l"(u64_of(b)));
    return f2_of(d);
}

}  // namespace gsph
