// RWKV-7 WKV forward with the blocks of a sequence side by side: what is left once wkv7_chunk.cu has walked every 64-token
// block from a zero state.  With S0 the state entering a block (row = value index i, column = key index j):
//     S_C = S0 diag(L_C) + S0 M' + U          y_t = R-_t S0^T + y'_t          sa_t = W~_t S0^T + sa'_t
// U, y', sa' being the zero-state results.  The first is a chain over the blocks (one CTA per sequence, the state in
// registers), the other two follow for all blocks at once.
//
// A sequence walked block after block takes 6.6 us per block, most of it work that does not depend on the state, and with
// fewer sequences than SMs the rest of the device idles meanwhile.  In this form a step of the chain takes 1.2-1.5 us (64
// mma.sync per warp behind one another's results) and the zero-state blocks fill the device: one sequence of 40 heads,
// T=2048, 224 -> 122 us; of 4 heads, T=4096, 407 -> 103 us.  M' is carried as high + low bf16 parts, U, y' and sa' in fp32, so
// that the split adds no rounding that the walk does not have in another place (errors against the oracle are the same).
//
// What a ring of CTAs does faster (see the rule in wkv7_chunk.cu) no longer comes here: long sequences of few heads stay, whose chain
// the start flags cut.
#include "common.cuh"
#include "tc05.cuh"
#include "chunk_common.cuh"
#include "device_once.cuh"
#include "wkv7_blocks.h"

namespace b200wkv {

int* wkv7_chunk_status_word();

namespace {

typedef __nv_bfloat16 bf;
using tc::cp_async16;
using tc::ldmatrix_x4;
using tc::ldmatrix_x4_trans;
using tc::mbar_arrive;
using tc::mma_bf16;

// ------------------------------------------------------------------ the chain --------
constexpr int kChainStages = 3;
constexpr int kUPitch = kC + 4;                 // float4 per column piece of U in shared memory: 64-bit reads hit 32 different banks
struct ChainStage {
    bf m[8][kC][8], m_low[8][kC][8];            // M'[j][j']: 8 column blocks of [64 rows j][8 columns j']
    float4 u[16][kUPitch];                      // U: 16 column pieces of [64 rows]
    float lam[kN];
};
struct ChainSmem {
    ChainStage st[kChainStages];
    uint64_t full[kChainStages], empty[kChainStages];
};
constexpr uint32_t kChainBytes = 2 * GTILE + 2 * GTILE + kN * 4;
static_assert(2 * (sizeof(ChainSmem) + 1024) <= 228 * 1024, "two CTAs per SM");

// One CTA per sequence: four warps with 16 rows of the state each, as mma.sync accumulator tiles, which are already in the
// register layout of the next product's left operand (as in wkv7_carry.cu), and a fifth that fetches the slots' tiles by bulk
// copies.  No warp waits for another one's rows.
//
// A slot with a start flag passes nothing of its entering state on (L_C = 0, M' = 0: the leaving state is U), so a sequence is
// offered to several CTAs ("pieces"): piece k starts behind the flagged slot nearest to k steps / pieces within half a piece of
// it, if there is one; every CTA finds the same cuts by itself, and one whose own cut does not exist has nothing to do.
__global__ void __launch_bounds__(160)
wkv7_chain_blocks_kernel(int Tlen, int H, int n_seq, int pieces, const uint32_t* __restrict__ length, const uint8_t* __restrict__ new_starts,
                         const bf* __restrict__ s0, const bf* __restrict__ mprime, const uint4* __restrict__ m_low,
                         const float4* __restrict__ u, const float* __restrict__ lam, unsigned char* __restrict__ s0_tiles,
                         size_t s0_stride, bf* __restrict__ s_out, float* __restrict__ s_at_len, int* __restrict__ status,
                         int* __restrict__ range_flag, int range_ticket) {
    let_next_in();
    if (word_behind(range_flag) == range_ticket) return;       // a decay outside the range: the call is redone

    extern __shared__ __align__(128) unsigned char smem[];
    ChainSmem& sm = *reinterpret_cast<ChainSmem*>(smem);
    const int bh = blockIdx.x % n_seq, piece = blockIdx.x / n_seq, bi = bh / H;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    const int i0 = warp * 16;
    const int L = min((int)length[bi], Tlen);
    const int nSlot = block_slots(Tlen), bl = L / kC;
    const bool cut = slot_tokens(nSlot - 1, Tlen, L).n > 0;
    const int steps = cut ? nSlot : nSlot - 1;
    auto slot_of = [&](int m) { return !cut || m <= bl ? m : m == bl + 1 ? nSlot - 1 : m - 1; };   // in order of time
    const size_t st_base = (size_t)bh * kN * kN, slot0 = (size_t)bh * nSlot;
    // the flagged step that cut k starts behind, or -1 (every warp by itself)
    auto find_cut = [&](int k) {
        const int target = (int)((long long)k * steps / pieces), half = steps / (2 * pieces);
        unsigned best = 0xffffffffu;
        for (int m = max(target - half, 0) + lane; m < min(target + half, steps - 1); m += 32)
            if (lam[(slot0 + slot_of(m)) * kN] == 0.f) best = min(best, (unsigned)(abs(m - target) * 2 + (m > target ? 1 : 0)) << 16 | (unsigned)m);
        best = __reduce_min_sync(0xffffffffu, best);
        return best == 0xffffffffu ? -1 : (int)(best & 0xffffu);
    };
    int first = 0, end = steps;                 // this CTA's steps; from a cut on, `first` only contributes U
    if (pieces > 1) {
        if (piece > 0 && (first = find_cut(piece)) < 0) return;
        for (int k = piece + 1; k < pieces; ++k) {
            const int c = find_cut(k);
            if (c >= 0) {
                end = c + 1;
                break;
            }
        }
    }
    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < kChainStages; ++i) {
            tc::mbar_init(&sm.full[i], 1);
            tc::mbar_init(&sm.empty[i], 4);
        }
        tc::mbar_init_fence();
    }
    __syncthreads();
    bool landed = true;
    if (warp == 4) {
        for (int m = first, it = 0; m < end; ++m, ++it) {
            const int stage = it % kChainStages;
            if (it >= kChainStages && !tc::mbar_wait(&sm.empty[stage], (it / kChainStages - 1) & 1)) {
                landed = false;                 // (the computing warps give up as well: nothing else is fetched)
                break;
            }
            ChainStage& s = sm.st[stage];
            uint64_t* bar = &sm.full[stage];
            const size_t slot = slot0 + slot_of(m);
            if (lane == 0) tc::mbar_expect_tx(bar, kChainBytes);
            __syncwarp();
            if (lane < 16) tc::bulk_load(&s.u[lane][0], u + slot * 1024 + lane * kC, kC * 16, bar);
            else if (lane == 16) tc::bulk_load(s.m, mprime + slot * (kN * kN), GTILE, bar);
            else if (lane == 17) tc::bulk_load(s.m_low, m_low + slot * 512, GTILE, bar);
            else if (lane == 18) tc::bulk_load(s.lam, lam + slot * kN, kN * 4, bar);
        }
        if (!landed && status != nullptr) atomicExch(status, 6);
        return;
    }
    float acc[8][4];                            // rows i0 + g, i0 + g + 8; column tile nt: columns 8 nt + 2q, + 1
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(s0 + st_base + (size_t)(i0 + g) * kN + nt * 8 + 2 * q));
        const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(s0 + st_base + (size_t)(i0 + g + 8) * kN + nt * 8 + 2 * q));
        acc[nt][0] = lo.x; acc[nt][1] = lo.y; acc[nt][2] = hi.x; acc[nt][3] = hi.y;
    }
    auto give_state = [&]() {
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const size_t at = st_base + (size_t)(i0 + g + 8 * hh) * kN + nt * 8 + 2 * q;
                *reinterpret_cast<uint32_t*>(s_out + at) = pack2(acc[nt][2 * hh], acc[nt][2 * hh + 1]);
                if (s_at_len != nullptr) *reinterpret_cast<float2*>(s_at_len + at) = make_float2(acc[nt][2 * hh], acc[nt][2 * hh + 1]);
            }
    };
    if (L == 0 && piece == 0) give_state();
    // whether a slot's first token is a start: its entering state is zero then
    const uint8_t* const ns_row = new_starts + (size_t)bi * Tlen;
    auto starts_anew = [&](int m) { return ns_row[slot_tokens(slot_of(min(m, steps - 1)), Tlen, L).p] != 0; };
    bool anew = starts_anew(first);
    for (int m = first, it = 0; m < end; ++m, ++it) {
        const int stage = it % kChainStages;
        const ChainStage& s = sm.st[stage];
        const int sl = slot_of(m);
        // the state entering the slot, in bf16: the left operand, and for the outputs (and the backward)
        uint32_t a[4][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            a[nt >> 1][(nt & 1) * 2] = pack2(acc[nt][0], acc[nt][1]);
            a[nt >> 1][(nt & 1) * 2 + 1] = pack2(acc[nt][2], acc[nt][3]);
        }
        if (!tc::mbar_wait(&sm.full[stage], (it / kChainStages) & 1)) {
            landed = false;
            break;
        }
        bool flagged = false;                   // (L_C is 0 in every channel then)
        float low[8][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const float2 l2 = *reinterpret_cast<const float2*>(&s.lam[nt * 8 + 2 * q]);
            if (nt == 0) flagged = l2.x == 0.f;
            const float4* const column = s.u[2 * nt + (q >> 1)];
            const float2 ulo = reinterpret_cast<const float2*>(column + i0 + g)[q & 1], uhi = reinterpret_cast<const float2*>(column + i0 + g + 8)[q & 1];
            acc[nt][0] = fmaf(acc[nt][0], l2.x, ulo.x);
            acc[nt][1] = fmaf(acc[nt][1], l2.y, ulo.y);
            acc[nt][2] = fmaf(acc[nt][2], l2.x, uhi.x);
            acc[nt][3] = fmaf(acc[nt][3], l2.y, uhi.y);
#pragma unroll
            for (int e = 0; e < 4; ++e) low[nt][e] = 0.f;
        }
        const int mi = lane >> 3, r8 = lane & 7;
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
#pragma unroll
            for (int np = 0; np < 4; ++np) {
                uint32_t b0, b1, b2, b3;        // column tiles 2 np (b0, b1) and 2 np + 1 (b2, b3)
                ldmatrix_x4_trans(b0, b1, b2, b3, &s.m[np * 2 + (mi >> 1)][ks * 16 + (mi & 1) * 8 + r8][0]);
                mma_bf16(acc[2 * np], a[ks], b0, b1);
                mma_bf16(acc[2 * np + 1], a[ks], b2, b3);
                ldmatrix_x4_trans(b0, b1, b2, b3, &s.m_low[np * 2 + (mi >> 1)][ks * 16 + (mi & 1) * 8 + r8][0]);
                mma_bf16(low[2 * np], a[ks], b0, b1);
                mma_bf16(low[2 * np + 1], a[ks], b2, b3);
            }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.empty[stage]);
        if (flagged) {                          // of a state that is no number, 0 x NaN has gone on (see wkv7_chunk.cu)
            bool odd = false;
#pragma unroll
            for (int e = 0; e < 16; ++e) odd |= (a[e >> 2][e & 3] & 0x7f80u) == 0x7f80u || (a[e >> 2][e & 3] & 0x7f800000u) == 0x7f800000u;
            if (odd) atomicExch(range_flag, range_ticket);
        }
        if (m > first || piece == 0) {
            unsigned char* const out = s0_tiles + (slot0 + sl) * s0_stride;
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                *reinterpret_cast<uint32_t*>(out + nt * GCB + (i0 + g) * 16 + 4 * q) = anew ? 0u : a[nt >> 1][(nt & 1) * 2];
                *reinterpret_cast<uint32_t*>(out + nt * GCB + (i0 + g + 8) * 16 + 4 * q) = anew ? 0u : a[nt >> 1][(nt & 1) * 2 + 1];
            }
        }
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[nt][e] += low[nt][e];
        anew = starts_anew(m + 1);
        const Slot tok = slot_tokens(sl, Tlen, L);
        if (tok.p + tok.n == L && (m > first || piece == 0)) give_state();
    }
    if (!landed && status != nullptr) atomicExch(status, 6);
}

// ------------------------------------------------------------------ the outputs --------
constexpr int kRowPitch = 72;                   // bf16 per row of R- and of the outputs (144 bytes)
struct OutSmem {
    bf s0[8][kN][8];                            // S0[i][j]: 8 column blocks of [64 rows i][8 columns j]
    bf w[8][kC][8];                             // W~[t][j], likewise
    bf rows[kC][kRowPitch];                     // R-[t][j], then the outputs
};

// One CTA of four warps per slot, each warp 16 tokens.  Bound by the traffic of its tiles (40 KB per slot, 80 KB with a
// residual), most of which the chain has just left in L2.
__global__ void __launch_bounds__(128)
wkv7_block_outputs_kernel(int Tlen, int H, int n_blk_slots, const uint32_t* __restrict__ length, const unsigned char* __restrict__ s0_tiles, size_t s0_stride,
                          const bf* __restrict__ rbar, BlockParts parts, unsigned char* __restrict__ saved, bf* __restrict__ y,
                          const int* __restrict__ range_flag, int range_ticket) {
    let_next_in();
    if (word_behind(range_flag) == range_ticket) return;
    __shared__ OutSmem sm;
    const int bh = blockIdx.x / n_blk_slots, sl = blockIdx.x % n_blk_slots, bi = bh / H, h = bh % H;
    const int L = min((int)length[bi], Tlen);
    const Slot tok = slot_tokens(sl, Tlen, L);
    if (tok.n <= 0) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3, mi = lane >> 3, r8 = lane & 7;
    const int t0 = warp * 16;
    const size_t slot = (size_t)bh * n_blk_slots + sl, tok_stride = (size_t)H * kN;
    const size_t base = ((size_t)bi * Tlen + tok.p) * tok_stride + (size_t)h * kN;
    const unsigned char* const tile = s0_tiles + slot * s0_stride;
#pragma unroll
    for (int c = tid; c < 512; c += 128) {
        const int t = c >> 3, piece = c & 7;
        cp_async16(reinterpret_cast<unsigned char*>(sm.s0) + c * 16, tile + c * 16, true);
        cp_async16(&sm.rows[t][piece * 8], rbar + base + (size_t)(t < tok.n ? t : 0) * tok_stride + piece * 8, t < tok.n);
        if (saved != nullptr) cp_async16(reinterpret_cast<unsigned char*>(sm.w) + c * 16, parts.w_tilde + slot * 512 + c, true);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    // an fp32 tile's rows t0 + g, + 8 and columns 8 nt + 2 q, + 1
    auto load_part = [&](const float4* tiles, float (*acc)[4]) {
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const float2 x = reinterpret_cast<const float2*>(tiles + slot * 1024 + (2 * nt + (q >> 1)) * 64 + t0 + g + 8 * hh)[q & 1];
                acc[nt][2 * hh] = x.x;
                acc[nt][2 * hh + 1] = x.y;
            }
    };
    float acc[8][4];
    load_part(parts.out, acc);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // acc[t][i] += A[t][j] S0[i][j]
    auto times_state = [&](auto left, float (*d)[4]) {
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
            uint32_t a[4];
            ldmatrix_x4(a[0], a[1], a[2], a[3], left(ks));
#pragma unroll
            for (int np = 0; np < 4; ++np) {
                uint32_t b0, b1, b2, b3;        // (tile 2 np: b0, b2), (tile 2 np + 1: b1, b3)
                ldmatrix_x4(b0, b1, b2, b3, &sm.s0[ks * 2 + (lane >> 4)][np * 16 + ((lane >> 3) & 1) * 8 + r8][0]);
                mma_bf16(d[2 * np], a, b0, b2);
                mma_bf16(d[2 * np + 1], a, b1, b3);
            }
        }
    };
    times_state([&](int ks) -> const void* { return &sm.rows[t0 + (mi & 1) * 8 + r8][16 * ks + (mi >> 1) * 8]; }, acc);
    __syncwarp();                               // (a warp reads and writes its own 16 rows only)
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        *reinterpret_cast<uint32_t*>(&sm.rows[t0 + g][nt * 8 + 2 * q]) = pack2(acc[nt][0], acc[nt][1]);
        *reinterpret_cast<uint32_t*>(&sm.rows[t0 + g + 8][nt * 8 + 2 * q]) = pack2(acc[nt][2], acc[nt][3]);
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = t0 + i * 4 + (lane >> 3), piece = lane & 7;
        if (t < tok.n) *reinterpret_cast<uint4*>(y + base + (size_t)t * tok_stride + piece * 8) = *reinterpret_cast<const uint4*>(&sm.rows[t][piece * 8]);
    }
    if (saved == nullptr) return;
    load_part(parts.sa, acc);
    times_state([&](int ks) -> const void* { return &sm.w[2 * ks + (mi >> 1)][t0 + (mi & 1) * 8 + r8][0]; }, acc);
    unsigned char* const out = saved + slot * kSavedBytes + (size_t)SAVED_SA * GTILE;
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        *reinterpret_cast<uint32_t*>(out + nt * GCB + (t0 + g) * 16 + 4 * q) = pack2(acc[nt][0], acc[nt][1]);
        *reinterpret_cast<uint32_t*>(out + nt * GCB + (t0 + g + 8) * 16 + 4 * q) = pack2(acc[nt][2], acc[nt][3]);
    }
}

}  // namespace

int wkv7_blocks_finish(cudaStream_t st, int B, int T, int H, const uint32_t* length, const uint8_t* ns, const void* s0, int* range_flag, int range_ticket,
                       const BlocksCall& c, void* y, void* s_out, float* s_at_len) {
    static DeviceOnce smem_attr;
    if (!smem_attr.ok([]() { return cudaFuncSetAttribute(wkv7_chain_blocks_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ChainSmem)); }))
        return B200WKV_ELAUNCH;
    // pieces: up to 8 of at least four steps
    const int quarter = block_slots(T) / 4, pieces = quarter < 1 ? 1 : quarter > 8 ? 8 : quarter;   // (steps fit 16 bits, see wkv7_blocks_bytes)
    if (launch_behind(wkv7_chain_blocks_kernel, B * H * pieces, 160, sizeof(ChainSmem), st, T, H, B * H, pieces, length, ns, (const bf*)s0, c.mprime, c.parts.m_low,
                                                                             c.parts.state, c.lam, c.s0_tiles, c.s0_stride, (bf*)s_out, s_at_len,
                      wkv7_chunk_status_word(), range_flag, range_ticket) != cudaSuccess)
        return B200WKV_ELAUNCH;
    const int nSlot = block_slots(T);
    return launch_behind(wkv7_block_outputs_kernel, B * H * nSlot, 128, 0, st, T, H, nSlot, length, c.s0_tiles, c.s0_stride, c.rbar, c.parts, c.saved,
                         (bf*)y, range_flag, range_ticket) == cudaSuccess ? B200WKV_OK : B200WKV_ELAUNCH;
}

}  // namespace b200wkv
