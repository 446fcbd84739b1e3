// extern "C" entry points declared in include/b200wkv.h: argument validation and dispatch.
#include <initializer_list>
#include "common.cuh"
#include "chunk_common.cuh"
#include "host_calls.h"
#include "wkv7_blocks.h"
#include "../../include/b200wkv_debug.h"

namespace b200wkv {
size_t wkv7_seq_residual_bytes(int B, int T, int H);
size_t wkv7_seq_carry_bytes(int B, int T, int H);
int wkv7_seq_fwd(cudaStream_t st, int dtype, int B, int T, int H, const void* w, const void* r, const void* k,
                 const void* v, const void* a, const void* b, const void* s0, const uint32_t* length,
                 const uint8_t* ns, void* y, void* s_out, void* residual, const int* run_if, int run_ticket,
                 int* residual_mark);
int wkv7_seq_bwd(cudaStream_t st, int dtype, int B, int T, int H, const void* w, const void* r, const void* k,
                 const void* v, const void* a, const void* b, const void* s0, const uint32_t* length,
                 const uint8_t* ns, const void* dy, const void* ds_out, void* residual, size_t residual_bytes, void* dw, void* dr,
                 void* dk, void* dv, void* da, void* db, void* ds0, const int* run_if);

// fp32 where wkv7_fp32_takes() says so: 16 tokens at a time (wkv7_fp32.cu)
bool wkv7_fp32_takes(int B, int T, int H);
size_t wkv7_fp32_workspace_bytes(int B, int T, int H);
size_t wkv7_fp32_kept_bytes(int B, int T, int H);
size_t wkv7_fp32_state_bytes(int B, int T, int H);
int wkv7_fp32_fwd(cudaStream_t st, int B, int T, int H, const void* w, const void* r, const void* k, const void* v, const void* a,
                  const void* b, const void* s0, const uint32_t* length, const uint8_t* ns, void* y, void* s_out, void* residual,
                  size_t residual_bytes, void* workspace);
int wkv7_fp32_bwd(cudaStream_t st, int B, int T, int H, const void* w, const void* r, const void* k, const void* v, const void* a,
                  const void* b, const uint32_t* length, const uint8_t* ns, const void* dy, const void* ds_out, void* residual,
                  size_t residual_bytes, void* workspace, void* dw, void* dr, void* dk, void* dv, void* da, void* db, void* ds0);

int wkv7_step(cudaStream_t st, int dtype, int B, int H, const void* w, const void* r, const void* k, const void* v,
              const void* a, const void* b, const void* s0, const uint32_t* length, const uint8_t* ns, void* y,
              void* s_out);
int wkv7_step_stream(cudaStream_t st, int dtype, int B, int H, const void* w, const void* r, const void* k, const void* v,
                     const void* a, const void* b, const void* s0, const uint32_t* length, const uint8_t* ns, void* y,
                     void* s_out, long long s_batch_stride);
int wkv7_step_stream_residency(int dtype, int* grid_per_sm, int* fit_per_sm);
size_t wkv7_chunk_residual_bytes(int B, int T, int H);
int wkv7_chunk_fwd(cudaStream_t st, int B, int T, int H, const void* w, const void* r, const void* k, const void* v,
                   const void* a, const void* b, const void* s0, const uint32_t* length, const uint8_t* ns, void* y,
                   void* s_out, void* residual, void* workspace, int* residual_mark, int** range_flag, int* range_ticket);
int wkv7_carry_bwd(cudaStream_t st, int B, int T, int H, const uint32_t* length, const void* dy,
                   const void* ds_out, void* residual, const int* residual_mark, void* ds0);
int wkv7_grad_bwd(cudaStream_t st, int B, int T, int H, const void* w, const void* r, const void* k, const void* v,
                  const void* a, const void* b, const uint32_t* length, const uint8_t* ns, const void* dy, void* residual,
                  const int* residual_mark, void* dw, void* dr, void* dk, void* dv, void* da, void* db);
int wkv7_chunk_status();

size_t wkv6_seq_residual_bytes(int B, int T, int H);
int wkv6_seq_fwd(cudaStream_t st, int dtype, int B, int T, int H, const void* r, const void* k, const void* v,
                 const void* w, int per_token, const void* u, const void* s0, const uint32_t* length,
                 const uint8_t* ns, void* y, void* s_out, void* residual, const int* run_if, int run_ticket,
                 int* residual_mark, const int* rest_of = nullptr);
int wkv6_seq_bwd(cudaStream_t st, int dtype, int B, int T, int H, const void* r, const void* k, const void* v,
                 const void* w, int per_token, const void* u, const uint32_t* length, const uint8_t* ns,
                 const void* dy, const void* ds_out, const void* residual, void* dr, void* dk, void* dv, void* dw,
                 void* du, void* ds0, const int* run_if, const int* rest_of = nullptr);
// A constant decay (versions 5, 5.2): fp32-accurate, run-parallel; `rest_of` above: their words per head, and only what these two left out is done
size_t wkv5_exact_partial_bytes(int B, int T, int H);
size_t wkv5_states_bytes(int B, int T, int H);
int* wkv5_odd_heads(int B, int T, int H, void* residual, void* workspace);
bool wkv5_exact_takes(int T, std::initializer_list<const void*> operands);
int wkv5_exact_fwd(cudaStream_t st, int B, int T, int H, const void* r, const void* k, const void* v, const void* w, const void* u,
                   const void* s0, const uint32_t* length, const uint8_t* ns, void* y, void* s_out, void* residual, int* residual_mark,
                   void* workspace);
int wkv5_exact_bwd(cudaStream_t st, int B, int T, int H, const void* r, const void* k, const void* v, const void* w, const void* u,
                   const uint32_t* length, const uint8_t* ns, const void* dy, const void* ds_out, void* residual, void* partial,
                   void* dr, void* dk, void* dv, void* dw, void* du, void* ds0);
size_t wkv6_chunk_residual_bytes(int B, int T, int H);
int wkv6_chunk_fwd(cudaStream_t st, int B, int T, int H, const void* r, const void* k, const void* v, const void* w,
                   int per_token, const void* u, const void* s0, const uint32_t* length, const uint8_t* ns, void* y,
                   void* s_out, void* residual, int* residual_mark, int** flag, int* ticket);
int wkv6_chunk_bwd(cudaStream_t st, int B, int T, int H, const void* r, const void* k, const void* v, const void* w,
                   const void* u, const uint32_t* length, const uint8_t* ns, const void* dy, const void* ds_out,
                   void* residual, const int* residual_mark, void* dr, void* dk, void* dv, void* dw, void* du, void* ds0);
size_t wkv4_residual_bytes(int B, int T, int C);
int wkv7_mix_partial_rows(int rows, int C);
int wkv7_mix_pre_fwd(cudaStream_t st, int dtype, int rows, int C, int use_vmix, const void* k, const void* wl, const void* al,
                     const void* v, const void* vf, const void* vl, const void* w0, const void* a0, const void* v0,
                     const void* k_k, const void* k_a, void* w, void* kp, void* vp, void* ai, void* bi);
int wkv7_mix_post_fwd(cudaStream_t st, int dtype, int rows, int C, float eps, const void* y, const void* r, const void* kp,
                      const void* vp, const void* g, const void* ln_w, const void* ln_b, const void* r_k, void* x);
int wkv7_mix_post_bwd(cudaStream_t st, int dtype, int rows, int C, float eps, const void* y, const void* r, const void* kp,
                      const void* vp, const void* g, const void* ln_w, const void* ln_b, const void* r_k, const void* gx, void* dy,
                      void* dr, void* dkp, void* dvp, void* dg, float* partial);
// The bf16 forward normally runs the chunked tensor-core kernel; a decay outside that kernel's range makes
// the token-sequential kernel behind it redo the call.  The last bytes of the residual tell the backward
// which of the two wrote it.
constexpr size_t kResidualMarkBytes = 16;
static int* residual_mark_of(void* residual, size_t bytes) {
    return residual ? reinterpret_cast<int*>(static_cast<char*>(residual) + bytes - kResidualMarkBytes) : nullptr;
}


// Whether all of these lie on boundaries of `bytes` (NULL does).  The kernels read and write vectors; an address that does not
// suit them is refused here, since a misaligned access ends the process's work on the device.
static bool aligned(size_t bytes, std::initializer_list<const void*> ps) {
    uintptr_t bits = 0;
    for (const void* p : ps) bits |= reinterpret_cast<uintptr_t>(p);
    return bits % bytes == 0;
}
// Whether `n` bytes at x and `m` bytes at y have any in common (NULL: none).
static bool meet(const void* x, size_t n, const void* y, size_t m) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(x), b = reinterpret_cast<uintptr_t>(y);
    return a != 0 && b != 0 && a < b + m && b < a + n;
}
// four elements, what the token-sequential kernels access at a time
static size_t vec4_bytes(int dtype) { return dtype == B200WKV_F32 ? 16 : 8; }

static int check_dims(int dtype, int B, int T, int H, int N) {
    if (dtype != B200WKV_F32 && dtype != B200WKV_BF16) return B200WKV_EDTYPE;
    if (B < 1 || T < 1 || H < 1 || N != kN) return B200WKV_ESHAPE;
    // element counts are indexed with size_t; the grid is B*H blocks
    if ((long long)B * H > 2147483647LL || (long long)B * T > 2147483647LL) return B200WKV_ESHAPE;   // token rows index tensor maps
    return B200WKV_OK;
}

// Whether a call with a residual takes 16 tokens at a time: where the residual has all the room, or keeps what it has to beside a
// workspace.  The forward and the backward of a residual have to agree on it (the host path sees to that: wkv7_kept_bytes).
static size_t fp32_full_bytes(int B, int T, int H) { return wkv7_fp32_kept_bytes(B, T, H) + wkv7_fp32_state_bytes(B, T, H); }
static bool wkv7_fp32_in_chunks(int B, int T, int H, size_t residual_bytes, const void* workspace) {
    return wkv7_fp32_takes(B, T, H) && residual_bytes >= (workspace != nullptr ? wkv7_fp32_kept_bytes(B, T, H) : fp32_full_bytes(B, T, H));
}

int wkv7_fwd(void* stream, int dtype, int B, int T, int H, int N, const void* w, const void* r, const void* k, const void* v,
             const void* a, const void* b, const void* s0, const uint32_t* length, const uint8_t* new_starts, void* y,
             void* s_out, void* residual, size_t residual_bytes, unsigned flags, void* workspace) {
    int st = check_dims(dtype, B, T, H, N);
    if (st != B200WKV_OK) return st;
    if (!w || !r || !k || !v || !a || !b || !s0 || !length || !new_starts || !y || !s_out) return B200WKV_ENULL;
    if (residual != nullptr && residual_bytes < b200wkv7_residual_min_bytes(dtype, B, T, H, N)) return B200WKV_ERESIDUAL;
    // one token and no residual wanted (recurrent decoding): a single pass over the state
    if (T == 1 && residual == nullptr) {
        if (!aligned(vec4_bytes(dtype), {w, r, k, v, a, b}) || !aligned(16, {s0, s_out})) return B200WKV_EUNSUPPORTED;
        return wkv7_step((cudaStream_t)stream, dtype, B, H, w, r, k, v, a, b, s0, length, new_starts, y, s_out);
    }
    const bool sequential = dtype == B200WKV_F32 || (flags & B200WKV_FLAG_SEQUENTIAL);
    if (!aligned(sequential ? vec4_bytes(dtype) : 16, {w, r, k, v, a, b, s0, y, s_out}) || !aligned(16, {residual, workspace}))
        return B200WKV_EUNSUPPORTED;
    if (!sequential) {
        int* mark = residual_mark_of(residual, b200wkv7_residual_bytes(dtype, B, T, H, N));
        int *range_flag = nullptr, ticket = 0;
        st = wkv7_chunk_fwd((cudaStream_t)stream, B, T, H, w, r, k, v, a, b, s0, length, new_starts, y, s_out, residual, workspace, mark,
                            &range_flag, &ticket);
        if (st != B200WKV_OK) return st;
        // does nothing unless the kernel above met a decay outside its range and left its ticket
        return wkv7_seq_fwd((cudaStream_t)stream, dtype, B, T, H, w, r, k, v, a, b, s0, length, new_starts, y, s_out, residual,
                            range_flag, ticket, mark);
    }
    if (dtype == B200WKV_F32 &&
        (residual != nullptr ? wkv7_fp32_in_chunks(B, T, H, residual_bytes, workspace) : workspace != nullptr))
        return wkv7_fp32_fwd((cudaStream_t)stream, B, T, H, w, r, k, v, a, b, s0, length, new_starts, y, s_out, residual, residual_bytes, workspace);
    return wkv7_seq_fwd((cudaStream_t)stream, dtype, B, T, H, w, r, k, v, a, b, s0, length, new_starts, y, s_out,
                        residual, nullptr, 0, nullptr);
}

int wkv7_bwd(void* stream, int dtype, int B, int T, int H, int N, const void* w, const void* r, const void* k, const void* v,
             const void* a, const void* b, const void* s0, const uint32_t* length, const uint8_t* new_starts, const void* dy,
             const void* ds_out, void* residual, size_t residual_bytes, void* dw, void* dr, void* dk, void* dv, void* da, void* db,
             void* ds0, unsigned flags, void* workspace) {
    int st = check_dims(dtype, B, T, H, N);
    if (st != B200WKV_OK) return st;
    if (!w || !r || !k || !v || !a || !b || !s0 || !length || !new_starts || !residual || !dw || !dr || !dk || !dv ||
        !da || !db || !ds0)
        return B200WKV_ENULL;
    if (residual_bytes < b200wkv7_residual_min_bytes(dtype, B, T, H, N)) return B200WKV_ERESIDUAL;
    const bool sequential = dtype == B200WKV_F32 || (flags & B200WKV_FLAG_SEQUENTIAL);
    if (!aligned(sequential ? vec4_bytes(dtype) : 16, {w, r, k, v, a, b, dy, dw, dr, dk, dv, da, db}) ||
        !aligned(vec4_bytes(dtype), {s0, ds_out, ds0}) || !aligned(16, {residual, workspace}))
        return B200WKV_EUNSUPPORTED;
    // must match the kernel family that filled the residual in b200wkv7_fwd (same dtype and flags)
    if (!sequential) {
        const int* mark = residual_mark_of(residual, b200wkv7_residual_bytes(dtype, B, T, H, N));
        // the sequential state-gradient carry, then the gradients of all blocks in parallel; the sequential kernels behind
        // them return at once unless the forward fell back to them
        st = wkv7_carry_bwd((cudaStream_t)stream, B, T, H, length, dy, ds_out, residual, mark, ds0);
        if (st != B200WKV_OK) return st;
        st = wkv7_grad_bwd((cudaStream_t)stream, B, T, H, w, r, k, v, a, b, length, new_starts, dy, residual, mark, dw, dr, dk, dv, da, db);
        if (st != B200WKV_OK) return st;
        return wkv7_seq_bwd((cudaStream_t)stream, dtype, B, T, H, w, r, k, v, a, b, s0, length, new_starts, dy, ds_out,
                            residual, b200wkv7_residual_bytes(dtype, B, T, H, N) - kResidualMarkBytes, dw, dr, dk, dv, da, db, ds0, mark);
    }
    // Gradients written over operands: the token-by-token kernels read a chunk's rows before they write them, where those for 16 tokens
    // at a time keep tiles in the gradients' buffers first.  ds0 over ds_out: without a carry between runs, which would be written
    // before the last read.  (The forward's checkpoints are the same for both.)
    bool in_place = false;
    const size_t stream_bytes = (size_t)B * T * H * kN * sizeof(float), state_bytes = (size_t)B * H * kN * kN * sizeof(float);
    if (dtype == B200WKV_F32) {
        for (const void* g : {dw, dr, dk, dv, da, db})
            for (const void* x : {w, r, k, v, a, b, dy}) in_place |= meet(g, stream_bytes, x, stream_bytes);
        if (meet(ds0, state_bytes, ds_out, state_bytes)) {
            in_place = true;
            residual_bytes = wkv7_seq_residual_bytes(B, T, H);
        }
    }
    if (dtype == B200WKV_F32 && !in_place && wkv7_fp32_in_chunks(B, T, H, residual_bytes, workspace))
        return wkv7_fp32_bwd((cudaStream_t)stream, B, T, H, w, r, k, v, a, b, length, new_starts, dy, ds_out, residual, residual_bytes, workspace, dw, dr,
                             dk, dv, da, db, ds0);
    return wkv7_seq_bwd((cudaStream_t)stream, dtype, B, T, H, w, r, k, v, a, b, s0, length, new_starts, dy, ds_out,
                        residual, residual_bytes, dw, dr, dk, dv, da, db, ds0, nullptr);
}

size_t wkv7_workspace_bytes(int dtype, int B, int T, int H, bool residual) {
    if (dtype == B200WKV_F32) return !residual ? wkv7_fp32_workspace_bytes(B, T, H) : wkv7_fp32_takes(B, T, H) ? wkv7_fp32_state_bytes(B, T, H) : 0;
    return wkv7_blocks_bytes(B, T, H, residual);
}
size_t wkv7_kept_bytes(int dtype, int B, int T, int H, bool workspace) {
    if (dtype != B200WKV_F32 || !wkv7_fp32_takes(B, T, H)) return b200wkv7_residual_bytes(dtype, B, T, H, kN);
    return workspace ? wkv7_fp32_kept_bytes(B, T, H) : b200wkv7_residual_min_bytes(dtype, B, T, H, kN);
}
size_t wkv7_bwd_workspace_bytes(int dtype, int B, int T, int H, size_t residual_bytes) {
    if (dtype != B200WKV_F32 || !wkv7_fp32_takes(B, T, H) || residual_bytes < wkv7_fp32_kept_bytes(B, T, H)) return 0;
    return residual_bytes < fp32_full_bytes(B, T, H) ? wkv7_fp32_state_bytes(B, T, H) : 0;
}

size_t wkv6_workspace_bytes(int dtype, bool per_token, int B, int T, int H) {
    if (dtype != B200WKV_BF16 || per_token) return 0;
    return wkv5_exact_takes(T, {}) ? wkv5_states_bytes(B, T, H) : 16;   // (16: the token-sequential kernels, which want no room)
}

int wkv6_fwd(void* stream, int dtype, int version, int B, int T, int H, int N, const void* r, const void* k,
                 const void* v, const void* w, const void* u, const void* s0, const uint32_t* length,
                 const uint8_t* new_starts, void* y, void* s_out, void* residual, size_t residual_bytes,
                 unsigned flags, void* workspace) {
    int st = check_dims(dtype, B, T, H, N);
    if (st != B200WKV_OK) return st;
    if (version != 5 && version != 6) return B200WKV_EUNSUPPORTED;
    if (!r || !k || !v || !w || !u || !s0 || !length || !new_starts || !y || !s_out) return B200WKV_ENULL;
    if (residual != nullptr && residual_bytes < b200wkv6_residual_bytes(dtype, B, T, H, N)) return B200WKV_ERESIDUAL;
    const bool sequential = dtype == B200WKV_F32 || (flags & B200WKV_FLAG_SEQUENTIAL);
    const bool exact = !sequential && version != 6 && (residual != nullptr || workspace != nullptr);      // wkv5_exact.cu, see below
    if (!aligned(sequential || exact ? vec4_bytes(dtype) : 16, {r, k, v, y}) || !aligned(version == 6 && !sequential ? 16 : vec4_bytes(dtype), {w}) ||
        !aligned(16, {residual, workspace}))
        return B200WKV_EUNSUPPORTED;
    if (dtype == B200WKV_BF16) {
        int* mark = residual_mark_of(residual, b200wkv6_residual_bytes(dtype, B, T, H, N));
        // With a constant decay (versions 5, 5.2) the decay's gradient is a sum over ALL tokens of per-token terms that
        // largely cancel; taken from bf16 tensor-core products it is only good to a few percent (10 % on short
        // sequences), so training calls of those versions take the fp32-accurate kernels of wkv5_exact.cu, with the
        // token-sequential ones for heads outside their domain (same checkpoints, marked as such) and for operands that the
        // wider accesses of the former do not suit.  So do calls without a residual that bring a workspace (the host path's,
        // which give the same bits with and without gradients).  Without either, and for everything of version 6: the
        // chunked kernels.
        if (exact && wkv5_exact_takes(T, {r, k, v, y, s0, s_out})) {
            st = wkv5_exact_fwd((cudaStream_t)stream, B, T, H, r, k, v, w, u, s0, length, new_starts, y, s_out, residual, mark, workspace);
            if (st != B200WKV_OK) return st;
            return wkv6_seq_fwd((cudaStream_t)stream, dtype, B, T, H, r, k, v, w, 0, u, s0, length, new_starts, y, s_out, residual, nullptr, 0,
                                mark, wkv5_odd_heads(B, T, H, residual, workspace));
        }
        if (exact && residual != nullptr &&     // the backward may take them all the same: no head is to be left out
            cudaMemsetAsync(wkv5_odd_heads(B, T, H, residual, nullptr), 0, (size_t)B * H * sizeof(int), (cudaStream_t)stream) != cudaSuccess)
            return B200WKV_ELAUNCH;
        if (sequential || exact)
            return wkv6_seq_fwd((cudaStream_t)stream, dtype, B, T, H, r, k, v, w, version == 6, u, s0, length, new_starts, y,
                                s_out, residual, nullptr, 0, mark);
        // the chunked tensor-core kernel, and behind it the sequential kernel, which runs only if the chunked one met
        // something outside its domain (it then redoes the whole call and marks the residual as its own)
        int* flag = nullptr;
        int ticket = 0;
        st = wkv6_chunk_fwd((cudaStream_t)stream, B, T, H, r, k, v, w, version == 6, u, s0, length, new_starts, y, s_out,
                            residual, mark, &flag, &ticket);
        if (st != B200WKV_OK) return st;
        return wkv6_seq_fwd((cudaStream_t)stream, dtype, B, T, H, r, k, v, w, version == 6, u, s0, length, new_starts, y,
                            s_out, residual, flag, ticket, mark);
    }
    return wkv6_seq_fwd((cudaStream_t)stream, dtype, B, T, H, r, k, v, w, version == 6, u, s0, length, new_starts, y,
                        s_out, residual, nullptr, 0, nullptr);
}
}  // namespace b200wkv

using namespace b200wkv;

extern "C" {

const char* b200wkv_strerror(int status) {
    switch (status) {
        case B200WKV_OK: return "ok";
        case B200WKV_EDTYPE: return "unsupported element type (expected B200WKV_F32 or B200WKV_BF16)";
        case B200WKV_ESHAPE: return "bad shape (every dimension must be >= 1 and the head size must be 64)";
        case B200WKV_ENULL: return "a required pointer is NULL";
        case B200WKV_ERESIDUAL: return "residual buffer is smaller than the size reported by *_residual_bytes";
        case B200WKV_ELAUNCH: return "CUDA kernel launch failed";
        case B200WKV_EUNSUPPORTED: return "combination not available in this build, or an operand's address does not suit the kernels' vector accesses";
        case B200WKV_ESCRATCH: return "problem exceeds the fixed built-in scratch area";
        case B200WKV_ESYMBOL: return "the built-in scratch area could not be materialised on this device (module load failed: out of device memory?)";
        default: return "unknown status";
    }
}

int b200wkv_abi_version(void) { return 2; }

int b200wkv_device_status(void) { return wkv7_chunk_status(); }

size_t b200wkv7_residual_min_bytes(int dtype, int B, int T, int H, int N) {
    if (check_dims(dtype, B, T, H, N) != B200WKV_OK) return 0;
    return dtype == B200WKV_F32 ? wkv7_seq_residual_bytes(B, T, H) : b200wkv7_residual_bytes(dtype, B, T, H, N);
}

size_t b200wkv7_residual_bytes(int dtype, int B, int T, int H, int N) {
    if (check_dims(dtype, B, T, H, N) != B200WKV_OK) return 0;
    // fp32 keeps a state every 16 tokens; bf16 uses the chunked tensor-core
    // kernels (a state every 64 tokens) unless B200WKV_FLAG_SEQUENTIAL asks otherwise, so size for both
    // (fp32: and for what the backward that works on all chunks side by side wants besides, where it does.  Where the sequences fill
    // their waves of CTAs it doesn't without a workspace: 36 KB per 16 tokens and head for 16 is more memory than the time is worth.)
    const size_t seq = wkv7_seq_residual_bytes(B, T, H);
    if (dtype == B200WKV_F32) {
        const size_t carry = wkv7_seq_carry_bytes(B, T, H);
        return carry != 0 && wkv7_fp32_takes(B, T, H) ? fp32_full_bytes(B, T, H) : seq + carry;
    }
    const size_t chk = wkv7_chunk_residual_bytes(B, T, H);
    // + one word at the end that says which of the two formats the forward left (see residual_mark_of)
    return (seq > chk ? seq : chk) + kResidualMarkBytes;
}

int b200wkv7_fwd(void* stream, int dtype, int B, int T, int H, int N, const void* w, const void* r, const void* k,
                 const void* v, const void* a, const void* b, const void* s0, const uint32_t* length,
                 const uint8_t* new_starts, void* y, void* s_out, void* residual, size_t residual_bytes,
                 unsigned flags) {
    return b200wkv::wkv7_fwd(stream, dtype, B, T, H, N, w, r, k, v, a, b, s0, length, new_starts, y, s_out, residual, residual_bytes, flags, nullptr);
}

int b200wkv7_bwd(void* stream, int dtype, int B, int T, int H, int N, const void* w, const void* r, const void* k,
                 const void* v, const void* a, const void* b, const void* s0, const uint32_t* length,
                 const uint8_t* new_starts, const void* dy, const void* ds_out, void* residual,
                 size_t residual_bytes, void* dw, void* dr, void* dk, void* dv, void* da, void* db, void* ds0,
                 unsigned flags) {
    return b200wkv::wkv7_bwd(stream, dtype, B, T, H, N, w, r, k, v, a, b, s0, length, new_starts, dy, ds_out, residual, residual_bytes, dw, dr, dk, dv, da,
                             db, ds0, flags, nullptr);
}

size_t b200wkv6_residual_bytes(int dtype, int B, int T, int H, int N) {
    if (check_dims(dtype, B, T, H, N) != B200WKV_OK) return 0;
    // fp32 uses the sequential kernels (an fp32 state every 16 tokens); bf16 uses the chunked tensor-core kernels (a
    // bf16 state every 16 tokens) with the sequential ones as their fallback, so size for both, plus one word at
    // the end that says which of the two formats the forward left
    size_t seq = wkv6_seq_residual_bytes(B, T, H);
    if (dtype == B200WKV_F32) return seq;
    const size_t chk = wkv6_chunk_residual_bytes(B, T, H);
    seq += wkv5_exact_partial_bytes(B, T, H);      // behind the checkpoints: the runs' shares of a constant decay's gradients
    return (seq > chk ? seq : chk) + kResidualMarkBytes;
}

int b200wkv6_fwd(void* stream, int dtype, int version, int B, int T, int H, int N, const void* r, const void* k,
                 const void* v, const void* w, const void* u, const void* s0, const uint32_t* length,
                 const uint8_t* new_starts, void* y, void* s_out, void* residual, size_t residual_bytes,
                 unsigned flags) {
    return b200wkv::wkv6_fwd(stream, dtype, version, B, T, H, N, r, k, v, w, u, s0, length, new_starts, y, s_out, residual, residual_bytes, flags, nullptr);
}

int b200wkv6_bwd(void* stream, int dtype, int version, int B, int T, int H, int N, const void* r, const void* k,
                 const void* v, const void* w, const void* u, const void* s0, const uint32_t* length,
                 const uint8_t* new_starts, const void* dy, const void* ds_out, void* residual,
                 size_t residual_bytes, void* dr, void* dk, void* dv, void* dw, void* du, void* ds0, unsigned flags) {
    int st = check_dims(dtype, B, T, H, N);
    if (st != B200WKV_OK) return st;
    if (version != 5 && version != 6) return B200WKV_EUNSUPPORTED;
    if (!r || !k || !v || !w || !u || !s0 || !length || !new_starts || !residual || !dr || !dk || !dv || !dw || !du || !ds0)
        return B200WKV_ENULL;
    if (residual_bytes < b200wkv6_residual_bytes(dtype, B, T, H, N)) return B200WKV_ERESIDUAL;
    if (!aligned(dtype == B200WKV_BF16 && version == 6 ? 16 : vec4_bytes(dtype), {r, k, v, dy, dr, dk, dv}) ||
        !aligned(dtype == B200WKV_BF16 && version == 6 ? 16 : vec4_bytes(dtype), {w}) || !aligned(vec4_bytes(dtype), {ds_out, ds0}) ||
        !aligned(16, {residual, dw, du}))
        return B200WKV_EUNSUPPORTED;
    if (dtype == B200WKV_BF16 && version != 6) {
        // (either family reads the checkpoints of the other)
        const bool sequential = (flags & B200WKV_FLAG_SEQUENTIAL) != 0 || !wkv5_exact_takes(T, {r, k, v, dy, dr, dk, dv});
        if (!sequential) {
            st = wkv5_exact_bwd((cudaStream_t)stream, B, T, H, r, k, v, w, u, length, new_starts, dy, ds_out, residual,
                                static_cast<char*>(residual) + wkv6_seq_residual_bytes(B, T, H), dr, dk, dv, dw, du, ds0);
            if (st != B200WKV_OK) return st;
        }
        return wkv6_seq_bwd((cudaStream_t)stream, dtype, B, T, H, r, k, v, w, 0, u, length, new_starts, dy, ds_out, residual, dr, dk, dv, dw, du,
                            ds0, nullptr, sequential ? nullptr : wkv5_odd_heads(B, T, H, residual, nullptr));
    }
    if (dtype == B200WKV_BF16) {
        // the forward's mark decides on the device which of the two runs; the other returns at once
        const int* mark = residual_mark_of(residual, b200wkv6_residual_bytes(dtype, B, T, H, N));
        st = wkv6_chunk_bwd((cudaStream_t)stream, B, T, H, r, k, v, w, u, length, new_starts, dy, ds_out,
                            residual, mark, dr, dk, dv, dw, du, ds0);
        if (st != B200WKV_OK) return st;
        return wkv6_seq_bwd((cudaStream_t)stream, dtype, B, T, H, r, k, v, w, 1, u, length, new_starts, dy, ds_out,
                            residual, dr, dk, dv, dw, du, ds0, mark);
    }
    return wkv6_seq_bwd((cudaStream_t)stream, dtype, B, T, H, r, k, v, w, version == 6, u, length, new_starts, dy,
                        ds_out, residual, dr, dk, dv, dw, du, ds0, nullptr);
}

size_t b200wkv4_residual_bytes(int dtype, int B, int T, int C) {
    if ((dtype != B200WKV_F32 && dtype != B200WKV_BF16) || B < 1 || T < 1 || C < 1) return 0;
    return wkv4_residual_bytes(B, T, C);
}

int b200wkv4_fwd(void* stream, int dtype, int B, int T, int C, const void* w, const void* u, const void* k,
                 const void* v, const void* s0, const uint32_t* length, const uint8_t* new_starts, void* s_out, void* y,
                 void* residual, size_t residual_bytes, unsigned flags) {
    if (dtype != B200WKV_F32 && dtype != B200WKV_BF16) return B200WKV_EDTYPE;
    if (B < 1 || T < 1 || C < 1 || (long long)B * C > 2147483647LL) return B200WKV_ESHAPE;
    if (!w || !u || !k || !v || !s0 || !length || !new_starts || !s_out || !y) return B200WKV_ENULL;
    if (residual != nullptr && residual_bytes < wkv4_residual_bytes(B, T, C)) return B200WKV_ERESIDUAL;
    (void)flags;
    return wkv4_fwd((cudaStream_t)stream, dtype, B, T, C, false, w, u, nullptr, k, v, s0, length, new_starts, s_out, y, residual);
}

int b200wkv4_bwd(void* stream, int dtype, int B, int T, int C, const void* w, const void* u, const void* k,
                 const void* v, const void* gy, const void* s0, const uint32_t* length, const uint8_t* new_starts,
                 const void* gs_new, const void* residual, size_t residual_bytes, void* gw, void* gu, void* gk,
                 void* gv, void* gs, unsigned flags) {
    if (dtype != B200WKV_F32 && dtype != B200WKV_BF16) return B200WKV_EDTYPE;
    if (B < 1 || T < 1 || C < 1 || (long long)B * C > 2147483647LL) return B200WKV_ESHAPE;
    if (!w || !u || !k || !v || !s0 || !length || !new_starts || !residual || !gw || !gu || !gk || !gv || !gs)
        return B200WKV_ENULL;
    if (residual_bytes < wkv4_residual_bytes(B, T, C)) return B200WKV_ERESIDUAL;
    (void)flags;
    return wkv4_bwd((cudaStream_t)stream, dtype, B, T, C, false, w, u, nullptr, k, v, gy, length, new_starts, gs_new, residual,
                    (float*)gw, (float*)gu, nullptr, gk, gv, gs);
}

int b200wkv7_step_inplace(void* stream, int dtype, int B, int H, int N, const void* w, const void* r, const void* k,
                          const void* v, const void* a, const void* b, void* state, long long state_batch_stride,
                          const uint32_t* length, const uint8_t* new_starts, void* y) {
    int st = check_dims(dtype, B, 1, H, N);
    if (st != B200WKV_OK) return st;
    if (!w || !r || !k || !v || !a || !b || !state || !y) return B200WKV_ENULL;
    const long long esz = dtype == B200WKV_F32 ? 4 : 2;
    if (state_batch_stride < (long long)H * N * N) return B200WKV_ESHAPE;
    const uintptr_t vec_bits = reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(r) | reinterpret_cast<uintptr_t>(k) |
                               reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b);
    if ((reinterpret_cast<uintptr_t>(state) & 31u) != 0 || (state_batch_stride * esz) % 32 != 0 || (vec_bits & 15u) != 0)
        return B200WKV_EUNSUPPORTED;
    return wkv7_step_stream((cudaStream_t)stream, dtype, B, H, w, r, k, v, a, b, state, length, new_starts, y, state,
                            state_batch_stride);
}

namespace {
int check_mix(int dtype, long long rows, int H, int N) {
    if (dtype != B200WKV_F32 && dtype != B200WKV_BF16) return B200WKV_EDTYPE;
    if (N != kN || H < 1 || H > 128 || rows < 1 || rows > 2147483647LL) return B200WKV_ESHAPE;
    return B200WKV_OK;
}
}  // namespace

int b200wkv7_mix_partial_rows(long long rows, int H, int N) {
    if (check_mix(B200WKV_F32, rows, H, N) != B200WKV_OK) return 0;
    return wkv7_mix_partial_rows((int)rows, H * N);
}

int b200wkv7_mix_pre_fwd(void* stream, int dtype, long long rows, int H, int N, int use_vmix, const void* k, const void* wl,
                         const void* al, const void* v, const void* v_first, const void* vl, const void* w0, const void* a0,
                         const void* v0, const void* k_k, const void* k_a, void* w, void* k_out, void* v_out, void* a_i,
                         void* b_i) {
    int st = check_mix(dtype, rows, H, N);
    if (st != B200WKV_OK) return st;
    if (!k || !wl || !al || !v || !w0 || !a0 || !k_k || !k_a || !w || !k_out || !v_out || !a_i || !b_i) return B200WKV_ENULL;
    if (use_vmix && (!v_first || !vl || !v0)) return B200WKV_ENULL;
    if (!aligned(16, {k, wl, al, v, v_first, vl, w0, a0, v0, k_k, k_a, w, k_out, v_out, a_i, b_i})) return B200WKV_EUNSUPPORTED;
    return wkv7_mix_pre_fwd((cudaStream_t)stream, dtype, (int)rows, H * N, use_vmix ? 1 : 0, k, wl, al, v, v_first, vl, w0, a0,
                            v0, k_k, k_a, w, k_out, v_out, a_i, b_i);
}

int b200wkv7_mix_pre_bwd(void* stream, int dtype, long long rows, int H, int N, int use_vmix, const void* k, const void* wl,
                         const void* al, const void* v, const void* v_first, const void* vl, const void* w0, const void* a0,
                         const void* v0, const void* k_k, const void* k_a, const void* gw, const void* gk_out,
                         const void* gv_out, const void* ga_i, const void* gb_i, void* dk, void* dwl, void* dal, void* dv,
                         void* dv_first, void* dvl, float* partial) {
    int st = check_mix(dtype, rows, H, N);
    if (st != B200WKV_OK) return st;
    if (!k || !wl || !al || !v || !w0 || !a0 || !k_k || !k_a || !gw || !gk_out || !gv_out || !ga_i || !gb_i || !dk || !dwl ||
        !dal || !dv || !partial)
        return B200WKV_ENULL;
    if (use_vmix && (!v_first || !vl || !v0 || !dv_first || !dvl)) return B200WKV_ENULL;
    if (!aligned(16, {k, wl, al, v, v_first, vl, w0, a0, v0, k_k, k_a, gw, gk_out, gv_out, ga_i, gb_i, dk, dwl, dal, dv, dv_first,
                    dvl, partial}))
        return B200WKV_EUNSUPPORTED;
    return wkv7_mix_pre_bwd((cudaStream_t)stream, dtype, (int)rows, H * N, use_vmix ? 1 : 0, k, wl, al, v, v_first, vl, w0, a0,
                            v0, k_k, k_a, gw, gk_out, gv_out, ga_i, gb_i, dk, dwl, dal, dv, dv_first, dvl, partial, MixPreExtra{});
}

int b200wkv7_mix_post_fwd(void* stream, int dtype, long long rows, int H, int N, float eps, const void* y, const void* r,
                          const void* k, const void* v, const void* g, const void* ln_w, const void* ln_b, const void* r_k,
                          void* x) {
    int st = check_mix(dtype, rows, H, N);
    if (st != B200WKV_OK) return st;
    if (!y || !r || !k || !v || !g || !ln_w || !ln_b || !r_k || !x) return B200WKV_ENULL;
    if (!aligned(16, {y, r, k, v, g, ln_w, ln_b, r_k, x})) return B200WKV_EUNSUPPORTED;
    return wkv7_mix_post_fwd((cudaStream_t)stream, dtype, (int)rows, H * N, eps, y, r, k, v, g, ln_w, ln_b, r_k, x);
}

int b200wkv7_mix_post_bwd(void* stream, int dtype, long long rows, int H, int N, float eps, const void* y, const void* r,
                          const void* k, const void* v, const void* g, const void* ln_w, const void* ln_b, const void* r_k,
                          const void* gx, void* dy, void* dr, void* dk, void* dv, void* dg, float* partial) {
    int st = check_mix(dtype, rows, H, N);
    if (st != B200WKV_OK) return st;
    if (!y || !r || !k || !v || !g || !ln_w || !ln_b || !r_k || !gx || !dy || !dr || !dk || !dv || !dg || !partial)
        return B200WKV_ENULL;
    if (!aligned(16, {y, r, k, v, g, ln_w, ln_b, r_k, gx, dy, dr, dk, dv, dg, partial})) return B200WKV_EUNSUPPORTED;
    return wkv7_mix_post_bwd((cudaStream_t)stream, dtype, (int)rows, H * N, eps, y, r, k, v, g, ln_w, ln_b, r_k, gx, dy, dr, dk,
                             dv, dg, partial);
}

int b200wkv_debug_step_residency(int dtype, int* grid_per_sm, int* fit_per_sm) {
    if (dtype != B200WKV_F32 && dtype != B200WKV_BF16) return B200WKV_EDTYPE;
    if (!grid_per_sm || !fit_per_sm) return B200WKV_ENULL;
    return wkv7_step_stream_residency(dtype, grid_per_sm, fit_per_sm);
}

int b200wkv_debug_wkv7_fwd_form(int sms, int largest_cluster, int B, int T, int H, int residual) {
    if (sms < 1 || check_dims(B200WKV_BF16, B, T, H, kN) != B200WKV_OK) return B200WKV_ESHAPE;
    return wkv7_fwd_form(sms, largest_cluster, B, T, H, residual != 0);
}

static int check_shift(int dtype, int B, int T, int D, int M) {
    if (dtype != B200WKV_F32 && dtype != B200WKV_BF16) return B200WKV_EDTYPE;
    if (B < 1 || T < 1 || D < 4 || (D % 4) != 0 || M < 1 || M > 8 || (long long)B * T > 2147483647LL || B > 65535) return B200WKV_ESHAPE;
    return B200WKV_OK;
}

namespace {
struct MixRows {   // the rows of a dense (M, D) array
    const void* p[8];
    MixRows(const void* mix, int dtype, int D, int M) {
        for (int m = 0; m < 8; ++m) p[m] = static_cast<const char*>(mix) + (size_t)(m < M ? m : 0) * D * (dtype == B200WKV_F32 ? 4 : 2);
    }
};
}  // namespace

int b200wkv_token_shift_fwd(void* stream, int dtype, int B, int T, int D, int M, const void* x, const void* prev,
                            const void* mix, const uint32_t* length, const uint8_t* new_starts, void* out,
                            void* state_out) {
    int st = check_shift(dtype, B, T, D, M);
    if (st != B200WKV_OK) return st;
    if (!x || !prev || !mix || !length || !new_starts || !out || !state_out) return B200WKV_ENULL;
    if (!aligned(dtype == B200WKV_F32 || D % 8 == 0 ? 16 : 8, {x, prev, mix, out, state_out})) return B200WKV_EUNSUPPORTED;
    const MixRows rows(mix, dtype, D, M);
    return token_shift_fwd((cudaStream_t)stream, dtype, B, T, D, M, x, prev, rows.p, length, new_starts, out, state_out);
}

int b200wkv_token_shift_bwd(void* stream, int dtype, int B, int T, int D, int M, const void* x, const void* prev,
                            const void* mix, const uint32_t* length, const uint8_t* new_starts, const void* gout,
                            const void* gstate, void* gx, void* gprev, void* gmix) {
    int st = check_shift(dtype, B, T, D, M);
    if (st != B200WKV_OK) return st;
    if (!x || !prev || !mix || !length || !new_starts || !gout || !gx || !gprev || !gmix) return B200WKV_ENULL;
    if (!aligned(dtype == B200WKV_F32 || D % 8 == 0 ? 16 : 8, {x, prev, mix, gout, gstate, gx, gprev}) || !aligned(16, {gmix}))
        return B200WKV_EUNSUPPORTED;
    const MixRows rows(mix, dtype, D, M);
    return token_shift_bwd((cudaStream_t)stream, dtype, B, T, D, M, x, prev, rows.p, length, new_starts, gout, gstate, gx,
                           gprev, gmix);
}

}  // extern "C"
