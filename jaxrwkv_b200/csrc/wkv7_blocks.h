// The block-parallel RWKV-7 forward (wkv7_blocks.cu): its workspace, and the launches behind the zero-state blocks.
#pragma once
#include "chunk_common.cuh"

namespace b200wkv {

// What the zero-state blocks leave per slot, all by rows of 16 bytes [column piece][row]: the state, the outputs and (with a
// residual) sa that follow from a zero entering state in fp32, the part of M' that its bf16 tile rounds off, and W~.
struct BlockParts {
    float4 *state, *out, *sa;
    uint4 *m_low, *w_tilde;
};
// Workspace of one call.  With a residual, M', R-, L_C and the entering states lie there; without one, here.
struct BlocksLayout {
    size_t state, out, m_low, sa, w_tilde, mprime, s0, rbar, lam, end;
};
inline BlocksLayout blocks_layout(int B, int T, int H, bool residual) {
    const size_t BH = (size_t)B * H, slots = BH * block_slots(T), none = 0;
    BlocksLayout l;
    l.state = 0;
    l.out = l.state + slots * 2 * GTILE;
    l.m_low = l.out + slots * 2 * GTILE;
    l.sa = l.m_low + slots * GTILE;
    l.w_tilde = l.sa + (residual ? slots * 2 * GTILE : none);
    l.mprime = l.w_tilde + (residual ? slots * GTILE : none);
    l.s0 = l.mprime + (residual ? none : slots * GTILE);
    l.rbar = l.s0 + (residual ? none : slots * GTILE);
    l.lam = l.rbar + (residual ? none : BH * (size_t)T * kN * 2);
    l.end = l.lam + (residual ? none : slots * kN * sizeof(float));
    return l;
}
// Where the pieces of a call lie; `saved` NULL: no residual.
struct BlocksCall {
    BlockParts parts;
    __nv_bfloat16 *mprime, *rbar;
    float* lam;
    unsigned char* s0_tiles;
    size_t s0_stride;
    unsigned char* saved;
};
// Bytes of workspace with which a call takes this form or a ring (0: neither), and which it is on a given device: 0 the walk, 1 this
// one, else a ring of so many CTAs
int wkv7_fwd_form(int sms, int largest, int B, int T, int H, bool residual);
size_t wkv7_blocks_bytes(int B, int T, int H, bool residual);
int wkv7_blocks_finish(cudaStream_t st, int B, int T, int H, const uint32_t* length, const uint8_t* ns, const void* s0, int* range_flag, int range_ticket,
                       const BlocksCall& call, void* y,
                       void* s_out, float* s_at_len);

}  // namespace b200wkv
