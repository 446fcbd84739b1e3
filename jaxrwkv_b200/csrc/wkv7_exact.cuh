// Shared by the fp32-arithmetic RWKV-7 kernels (wkv7_chain.cu, wkv7_seq.cu, wkv7_fp32.cu).
#pragma once
#include "common.cuh"

namespace b200wkv {

constexpr int kExactChunk = 16;   // tokens per staged chunk == spacing of the saved state checkpoints

// two fp32 values in a 64-bit register: fma.rn.f32x2 rounds each as fmaf does
struct Pair { unsigned long long u; };
__device__ __forceinline__ Pair pair(float a, float b) {
    Pair p;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p.u) : "f"(a), "f"(b));
    return p;
}
__device__ __forceinline__ float2 unpack(Pair p) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(p.u));
    return f;
}
__device__ __forceinline__ Pair fma2(Pair a, Pair b, Pair c) {
    Pair d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d.u) : "l"(a.u), "l"(b.u), "l"(c.u));
    return d;
}
__device__ __forceinline__ Pair mul2(Pair a, Pair b) {
    Pair d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d.u) : "l"(a.u), "l"(b.u));
    return d;
}
__device__ __forceinline__ Pair add2(Pair a, Pair b) {
    Pair d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d.u) : "l"(a.u), "l"(b.u));
    return d;
}
__device__ __forceinline__ float4 decay4(float4 w) {
    return make_float4(expf(-expf(w.x)), expf(-expf(w.y)), expf(-expf(w.z)), expf(-expf(w.w)));
}

}  // namespace b200wkv
