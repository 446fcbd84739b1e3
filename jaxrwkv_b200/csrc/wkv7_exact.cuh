// Shared by the fp32-arithmetic RWKV-7 kernels (wkv7_chain.cu, wkv7_seq.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200wkv {

constexpr int kExactChunk = 16;   // tokens per staged chunk == spacing of the saved state checkpoints

}  // namespace b200wkv
