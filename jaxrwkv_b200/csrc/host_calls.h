// Calls of libb200wkv.so that its own host path (host_ext.cpp) makes beyond the C ABI: fused forms of an operator for
// which the reference has no custom call.  Plain C++ linkage: not part of the boundary that other hosts bind.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200wkv {

// RWKV-4 with the receptance product inside (y = r * wkv; r NULL: without) and, with `raw_w`, the decay parameter w
// before -exp().  The backward writes dr when r is given, and per-sequence sums of dw' and du (B, C).
int wkv4_fwd(cudaStream_t st, int dtype, int B, int T, int C, bool raw_w, const void* w, const void* u, const void* r, const void* k,
             const void* v, const void* s0, const uint32_t* length, const uint8_t* ns, void* s_out, void* y, void* residual);
int wkv4_bwd(cudaStream_t st, int dtype, int B, int T, int C, bool raw_w, const void* w, const void* u, const void* r, const void* k,
             const void* v, const void* gy, const uint32_t* length, const uint8_t* ns, const void* gs_new,
             const void* residual, float* gw, float* gu, void* gr, void* gk, void* gv, void* gs);
// dw = -exp(w) * sum_b gw, du = sum_b gu, in the element type
int wkv4_parameter_grads(cudaStream_t st, int dtype, int B, int C, const void* w, const float* gw, const float* gu, void* dw, void* du);

}  // namespace b200wkv
