// Calls of libb200wkv.so that its own host path (host_ext.cpp) makes beyond the C ABI: fused forms of an operator for
// which the reference has no custom call.  Plain C++ linkage: not part of the boundary that other hosts bind.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200wkv {

// b200wkv7_fwd with a workspace of wkv7_workspace_bytes() (0: the call wants none, workspace NULL).
size_t wkv7_workspace_bytes(int dtype, int B, int T, int H, bool residual);
int wkv7_fwd(void* stream, int dtype, int B, int T, int H, int N, const void* w, const void* r, const void* k, const void* v,
             const void* a, const void* b, const void* s0, const uint32_t* length, const uint8_t* new_starts, void* y,
             void* s_out, void* residual, size_t residual_bytes, unsigned flags, void* workspace);

// b200wkv7_bwd with a workspace of wkv7_bwd_workspace_bytes() (0: it wants none, NULL).
size_t wkv7_bwd_workspace_bytes(int dtype, int B, int T, int H, size_t residual_bytes);
int wkv7_bwd(void* stream, int dtype, int B, int T, int H, int N, const void* w, const void* r, const void* k, const void* v,
             const void* a, const void* b, const void* s0, const uint32_t* length, const uint8_t* new_starts, const void* dy,
             const void* ds_out, void* residual, size_t residual_bytes, void* dw, void* dr, void* dk, void* dv, void* da, void* db,
             void* ds0, unsigned flags, void* workspace);
// What is to be kept for the backward (N = 64) where the forward has its workspace or, where it wants one, doesn't.  The size tells the
// backward which kernels filled it.
size_t wkv7_kept_bytes(int dtype, int B, int T, int H, bool workspace);

// b200wkv6_fwd; a call without a residual may bring a workspace of wkv6_workspace_bytes() (0: it wants none, NULL) and then has
// the arithmetic of a call with one.
size_t wkv6_workspace_bytes(int dtype, bool per_token, int B, int T, int H);
int wkv6_fwd(void* stream, int dtype, int version, int B, int T, int H, int N, const void* r, const void* k, const void* v,
             const void* w, const void* u, const void* s0, const uint32_t* length, const uint8_t* new_starts, void* y,
             void* s_out, void* residual, size_t residual_bytes, unsigned flags, void* workspace);

// dw and du of operands shared by the batch (C channels) in the element type, from b200wkv6_bwd's sums per sequence; directly behind it in
// the stream.  gw NULL: du alone
int wkv6_parameter_grads(cudaStream_t st, int dtype, int B, int C, const float* gw, const float* gu, void* dw, void* du);

// RWKV-4 with the receptance product inside (y = r * wkv; r NULL: without) and, with `raw_w`, the decay parameter w
// before -exp().  The backward writes dr when r is given, and per-sequence sums of dw' and du (B, C).
int wkv4_fwd(cudaStream_t st, int dtype, int B, int T, int C, bool raw_w, const void* w, const void* u, const void* r, const void* k,
             const void* v, const void* s0, const uint32_t* length, const uint8_t* ns, void* s_out, void* y, void* residual);
int wkv4_bwd(cudaStream_t st, int dtype, int B, int T, int C, bool raw_w, const void* w, const void* u, const void* r, const void* k,
             const void* v, const void* gy, const uint32_t* length, const uint8_t* ns, const void* gs_new,
             const void* residual, float* gw, float* gu, void* gr, void* gk, void* gv, void* gs);
// dw = -exp(w) * sum_b gw, du = sum_b gu, in the element type
int wkv4_parameter_grads(cudaStream_t st, int dtype, int B, int C, const void* w, const float* gw, const float* gu, void* dw, void* du);


// The token shift with the M rows of mix coefficients where the model keeps them (M <= 8).
int token_shift_fwd(cudaStream_t st, int dtype, int B, int T, int D, int M, const void* x, const void* prev,
                    const void* const* mix, const uint32_t* length, const uint8_t* ns, void* out, void* state_out);
int token_shift_bwd(cudaStream_t st, int dtype, int B, int T, int D, int M, const void* x, const void* prev,
                    const void* const* mix, const uint32_t* length, const uint8_t* ns, const void* gout, const void* gstate,
                    void* gx, void* gprev, void* gmix);
// The backward of the stage in front of the operator with what else meets there: more cotangents of k' and v' (gkp2, gvp2) and
// of the first layer's v (gv_out), and r's second share (gr += dr).  NULL: none.
struct MixPreExtra {
    const void *gkp2, *gvp2, *gv_out, *dr;
    void* gr;
};
int wkv7_mix_pre_bwd(cudaStream_t st, int dtype, int rows, int C, int use_vmix, const void* k, const void* wl, const void* al,
                     const void* v, const void* vf, const void* vl, const void* w0, const void* a0, const void* v0,
                     const void* k_k, const void* k_a, const void* gw, const void* gkp, const void* gvp, const void* gai,
                     const void* gbi, void* dk, void* dwl, void* dal, void* dv, void* dvf, void* dvl, float* partial,
                     const MixPreExtra& extra);
// y == NULL: x = act(x) in place; else x *= act'(.) in terms of y = act(.)
enum { kTanh = 1, kSigmoid = 2 };
int activation(cudaStream_t st, int dtype, int act, long long n, void* x, const void* y);
// The column sums of up to three arrays of partial rows, one behind the other into `out` in the element type (columns: a
// multiple of 32 each).
struct PartialRows {
    const float* partial;
    int rows, cols;
};
int column_sums(cudaStream_t st, int dtype, const PartialRows (&of)[3], void* out);

}  // namespace b200wkv
