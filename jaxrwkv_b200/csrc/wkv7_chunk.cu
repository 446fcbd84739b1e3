// RWKV-7 WKV forward, chunked along T on the Blackwell tensor cores (bf16 I/O, fp32 state).
//
// One CTA (256 threads) per (batch, head) walks the sequence in chunks of up to 64 tokens.  With
// L_t = prod_{s<=t} decay_s (per key channel, inside the chunk) and the scaled operands
//   A~_t = a_t * L_{t-1}   R~_t = r_t * L_t   B~_t = b_t / L_t   K~_t = k_t / L_t
//   B^_t = b_t * L_C / L_t K^_t = k_t * L_C / L_t                (L_C = decay over the whole chunk)
// the recurrence  S <- S diag(decay) + (S a) b^T + v k^T,  y = S r  becomes, for a chunk entered
// with state S0 (row = value index, column = key index):
//   [A_ab A_ak; P_rb P_rk] = [A~; R~] [B~; K~]^T            strictly / inclusively lower triangular
//   G   = A_ak V + A~ S0^T                                  (token x value)
//   sa  = (I - A_ab)^-1 G                                   row t is S_{t-1} a_t
//   Y   = P_rk V + R~ S0^T + P_rb sa
//   S_C = S0 diag(L_C) + sa^T B^ + V^T K^
// All products are tcgen05.mma (M=128, bf16 operands from shared memory, fp32 accumulators in
// TMEM); the unit-triangular inverse is an fp32 forward substitution on CUDA cores; the state
// stays in TMEM in fp32 for the whole sequence.
//
// A start flag on a token of the chunk cuts every dependence of the tokens from it on, on what came before: the pairwise
// products lose the columns in front of the row's last flag, the S0 products the rows from the first flag on, B^ and K^
// the rows in front of the last flag, and the decayed entering state is dropped.  (Ending the chunk in front of every
// flag instead, as an earlier form did, costs a whole chunk's time per flag, and a backward that can follow it: forward and
// backward at B=6, T=2043, H=32 with a flag every 512 tokens took 970-990 us so, and take 676 us with the masks, while
// a forward without flags, B=8, T=4096, H=32, takes 595 us in that form and 594-597 with the masks.)  The
// cumulative decay is not restarted: only ratios inside a segment survive the masks.  A chunk ends early only where the
// state is wanted, at `length`, and at the end of the sequence; the rows behind its end are zero.
//
// Data movement: the raw rows of the next chunk arrive in shared memory by tiled bulk copies
// (cp.async.bulk.tensor) while the current chunk finishes.  When a residual is requested, every chunk
// leaves bf16 operand slabs for the backward (T, A_ak, P_rb, P_rk, sa, S0; most of them by bulk stores out of shared
// memory) so that the backward need not recompute them.
//
// Semantics: BaseRWKV.inner_loop of jaxrwkv (src/jaxrwkv/rwkv7.py:199-220).
#include "common.cuh"
#include "tc05.cuh"
#include "chunk_common.cuh"
#include "tmap.cuh"
#include "wkv7_blocks.h"

#include <algorithm>
#include <atomic>

namespace b200wkv {

namespace {

// shared-memory map (bytes); two CTAs per SM
constexpr int OFF_AR = 0;                        // [A~ ; R~]           128-row slab  } dead once the first
constexpr int OFF_BK = OFF_AR + SLAB128;         // [B~ ; K~]           128-row slab  } products are done:
constexpr int OFF_S0 = OFF_BK + SLAB128;         // S0 in bf16          64-row slab   } LF, X, SCR alias them
constexpr int OFF_BH = OFF_S0 + SLAB64;          // B^                  64-row slab
constexpr int OFF_KH = OFF_BH + SLAB64;          // K^                  64-row slab
constexpr int OFF_SA = OFF_KH + SLAB64;          // sa                  64-row slab   } consecutive: the MN-major
constexpr int OFF_V = OFF_SA + SLAB64;           // V                   64-row slab   } A operands of the state
constexpr int OFF_M2A = OFF_V + SLAB64;          // [A_ak ; P_rk]       128-row slab  } update span two slabs
constexpr int OFF_G = OFF_M2A;                   // G (aliases M2A once the A_ak/P_rk product is done)
constexpr int OFF_TP = OFF_M2A + SLAB128;        // [Tinv ; P_rb]       128-row slab   (CUM aliases TP)
constexpr int OFF_SMALL = OFF_TP + LF_PITCH * 64 * 4;   // TP is 16512 B; the scan buffer that aliases it needs 17408
constexpr int OFF_LF = OFF_AR;                           // fp32 A_ab
constexpr int OFF_X = OFF_LF + LF_PITCH * 64 * 4;        // fp32 (I - A_ab)^-1
constexpr int OFF_SCR = OFF_X + LF_PITCH * 64 * 4;       // scratch of the inverse
constexpr int OFF_CUM = OFF_TP;
// Result tiles of a chunk, written by the last epilogue over slabs whose products are done and that no copy to the
// residual reads (V, and G = W~), and sent to global memory by bulk copies: the 64 output rows as [64][128 bytes]
// with the 128-byte swizzle of the tiled copy (piece index XOR row mod 8), and M' as 8 column blocks of [64 rows]
// [16 bytes], the layout of the saved tiles.
constexpr int OFF_YT = (OFF_V + 1023) / 1024 * 1024;
constexpr int OFF_MT = OFF_YT + kC * kN * 2;
constexpr int OFF_RT = (OFF_BH + 1023) / 1024 * 1024;   // P_rb W~ (token rows, swizzled like the outputs) over B^, K^
static_assert(OFF_RT + kC * kN * 2 <= OFF_SA, "the P_rb W~ tile must lie over B^ and K^");
static_assert(OFF_MT + GTILE <= OFF_M2A + SLAB64, "result tiles must lie over V and G");
// Staging tiles for the raw rows of the NEXT chunk (6 streams x 64 tokens x 128 bytes), filled by tiled
// bulk copies once the inverse is done: tiles 0..4 over AR + BK + S0, tile 5 over the P_rk half of M2A.
constexpr int STG_TILE = kC * kN * 2;
static_assert(5 * STG_TILE <= 2 * SLAB128 + SLAB64 && STG_TILE <= SLAB128 - SLAB64, "staging tiles must fit their hosts");
__device__ __forceinline__ int stage_off(int m) { return m < 5 ? OFF_AR + m * STG_TILE : OFF_M2A + SLAB64; }
// A ring's step once the zero-state products are done (nothing here lies over the staging tiles):
constexpr int OFF_IN = OFF_BH;                   // the entering state, fp32, 16 column pieces of [64 rows][16 bytes], written by the CTA in front
constexpr int OFF_SB = OFF_SA;                   // the same in bf16         64-row slab
constexpr int OFF_MH = OFF_V;                    // M', its bf16 part        64-row slab
constexpr int OFF_ML = OFF_G;                    // M', what that rounds off 64-row slab (over W~)
constexpr int OFF_WR = OFF_TP;                   // [W~ ; R-]                128-row slab
// ... of kExactRingForm: [W~ ; R~], without a residual [P_rb W~ ; R~], and
constexpr int OFF_PW = OFF_ML;                   // with one P_rb W~         64-row slab, once the state products are done
static_assert(OFF_IN + kN * kN * 4 <= OFF_SB, "the entering state lies over B^ and K^");
struct Small {
    float h1[kN];        // cumulative log-decay of tokens 0..31, stored [e][jb] for channel 8 jb + e
    float tot[kN];       // ... of the whole chunk
    float lam[kN];       // exp(tot)
    float lamt[kN];      // the same, stored [e][jb]
    uint64_t bar[5];   // 0..3 product rounds, 4 staging tiles
    uint64_t ring[4];  // a ring's: state products, output products, the entering state has arrived, the next CTA is ready for one
    uint32_t nsm[2];
    uint32_t tmem;
};
constexpr int SMEM_BYTES = OFF_SMALL + (int)sizeof(Small);
static_assert(OFF_SCR + TRI_SCR_FLOATS * 4 <= OFF_BH, "inverse work space must fit over AR+BK+S0");
static_assert(2 * (SMEM_BYTES + 1024) <= 228 * 1024, "two CTAs per SM");

// What only chunks with start flags and chunks of fewer than 64 tokens need is kept out of the walk's loop: the passes over TMEM
// are functions that are not inlined, and the flags are read back from shared memory where a flagged chunk needs them.  With the
// passes inlined and the flags' 64 bits live across the loop body, every chunk WITHOUT flags paid 1 % (forward with a residual at
// B=8, T=4096, H=32: 603-607 -> 594-597 us; without a residual 543 -> 531; B=6, T=2043 with a flag every 512 tokens 321 -> 318).  A second copy of the loop body for full chunks without flags is no faster on such sequences and
// loses where both kinds mix, the two bodies evicting each other's instructions (B=8, T=1024, H=32, a flag every 100 tokens: 200 us
// against 178).
__device__ __forceinline__ uint64_t start_mask(const Small& sm) {   // bit t: a flag on token t of the chunk
    const volatile uint32_t* m = sm.nsm;
    return (uint64_t)m[0] | ((uint64_t)m[1] << 32);
}
__device__ __forceinline__ bool in_first(uint64_t mask, int t) { return (mask & ((2ull << t) - 1ull)) == 0; }   // no flag at or before token t
__device__ __forceinline__ bool in_last(uint64_t mask, int t) { return ((mask >> t) >> 1) == 0; }               // none behind it
// 64 columns of the pairwise products in TMEM, row t: nothing from in front of the row's last flag
__device__ __noinline__ void mask_pairs(uint32_t taddr, uint64_t mask, int t) {
    const uint64_t upto = mask & ((2ull << t) - 1ull);
    const int from = upto != 0 ? 63 - __clzll((long long)upto) : 0;
#pragma unroll
    for (int part = 0; part < 2; ++part) {
        float x[32];
        tc::tmem_ld32(taddr + part * 32, x);
        tc::tmem_wait_ld();
#pragma unroll
        for (int s = 0; s < 32; ++s) x[s] = s + part * 32 >= from ? x[s] : 0.f;
        tc::tmem_st32(taddr + part * 32, x);
    }
    tc::tmem_wait_st();
}
// 32 columns of the S0 products, row t: nothing from the first flag on
__device__ __noinline__ void mask_state_products(uint32_t taddr, uint64_t mask, int t) {
    float g[32];
    tc::tmem_ld32(taddr, g);
    tc::tmem_wait_ld();
    const bool first = in_first(mask, t);
#pragma unroll
    for (int c = 0; c < 32; ++c) g[c] = first ? g[c] : 0.f;
    tc::tmem_st32(taddr, g);
    tc::tmem_wait_st();
}
// The masks put zeros where a start flag cuts, and the products that follow multiply them: 0 x NaN would carry what is not
// a number over the flag.  So a flagged chunk that meets any in k, v, a, b or its entering state leaves the call to the
// token-sequential kernel, which drops the state at a flag whatever it is.  (The walk looks at the operands in registers; blocks
// side by side, whose body that costs 4 us of 57, at what came of them.)  The sums stay 0 for numbers and are NaN otherwise.
__device__ __forceinline__ void add_odd(__nv_bfloat162& sum, const uint4& x) {
    const __nv_bfloat162 zero = __floats2bfloat162_rn(0.f, 0.f);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&x);
#pragma unroll
    for (int i = 0; i < 4; ++i) sum = __hfma2(h[i], zero, sum);
}
__device__ __forceinline__ bool is_odd(const __nv_bfloat162& sum) { return __low2float(sum) + __high2float(sum) != 0.f; }
// this thread's 32 columns of a row of sa, W~ and V in their slabs
__device__ __noinline__ void leave_to_sequential_if_odd(const unsigned char* sa, const unsigned char* w_tilde, const unsigned char* v, int* range_flag,
                                                        int range_ticket) {
    __nv_bfloat162 odd = __floats2bfloat162_rn(0.f, 0.f);
    for (const unsigned char* row : {sa, w_tilde, v})
#pragma unroll
        for (int c = 0; c < 4; ++c) add_odd(odd, *reinterpret_cast<const uint4*>(row + c * CB64));
    if (is_odd(odd)) atomicExch(range_flag, range_ticket);
}
// 32 columns in TMEM added in fp32 onto a bf16 row in global memory; the whole warp calls it
__device__ __noinline__ void add_to_row(uint32_t taddr, __nv_bfloat16* row, bool live) {
    float m[32];
    tc::tmem_ld32(taddr, m);
    tc::tmem_wait_ld();
    if (!live) return;
    uint4* to = reinterpret_cast<uint4*>(row);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        float x[8];
        unpack8(to[c], x);
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] += m[c * 8 + e];
        to[c] = pack8(x);
    }
}

// four K=16 steps (64 deep) of D (+)= A B
__device__ __forceinline__ void mma_k64(uint32_t d, Op a, Op b, uint32_t idesc, bool accumulate) {
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) tc::mma(d, op_desc(a, ks), op_desc(b, ks), idesc, accumulate || ks > 0);
}

__device__ int g_status;  // last device-side error (0 = none); see wkv7_chunk_status()


// 32 columns of one row of an fp32 tile [16 column pieces][64 rows] (of four columns): a warp's rows are contiguous
__device__ __forceinline__ void store_part(float4* tiles, size_t slot, int hsel, int row, const float* x) {
#pragma unroll
    for (int c = 0; c < 8; ++c) tiles[slot * 1024 + (hsel * 8 + c) * 64 + row] = make_float4(x[c * 4], x[c * 4 + 1], x[c * 4 + 2], x[c * 4 + 3]);
}

__device__ __forceinline__ void load_part(const float4* tiles, size_t slot, int hsel, int row, float* x) {
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const float4 v = tiles[slot * 1024 + (hsel * 8 + c) * 64 + row];
        x[c * 4] = v.x; x[c * 4 + 1] = v.y; x[c * 4 + 2] = v.z; x[c * 4 + 3] = v.w;
    }
}

// kWalk: a CTA walks one sequence (or piece of one).  The others do everything of a block that does not depend on the entering
// state S0 as if that were zero, which leaves, with U, y', sa' the zero-state results,
//     S_C = S0 diag(L_C) + S0 M' + U          y_t = R-_t S0^T + y'_t          sa_t = W~_t S0^T + sa'_t,
// M' as high + low bf16 parts and U, y', sa' in fp32, so that the split adds no rounding that the walk does not have elsewhere.
// kBlocks: the blocks of all sequences as one list, a CTA has consecutive ones, and what depends on S0 is left to the kernels of
// wkv7_blocks.cu.
// kRing: a cluster of CTAs walks one sequence, whose blocks are dealt out in turn.  A CTA takes S0 out of its shared memory, where
// the CTA with the block in front has put it, passes S_C on to the next one and then finishes its outputs.  A state's way through a
// CTA takes 2700 cycles (330 to the operand slab, 870 products, 400 results, 1000 to the next CTA), a block 17 k of its CTA's, 13 k of
// them before the state is needed.  One sequence of 40 heads, T=1999: 114 us in kBlocks, 83 by rings of six; 80 sequences,
// T=1024: 111 walked, 99 by rings of three (kExactRing).
// R- = R~ + P_rb W~ is rounded once more than R~ and sa are before they meet in the walk, which makes the outputs' errors 0.15 % larger
// than the walk's (4.090e-3 of them against 4.084e-3, 80 sequences, T=1000), in blocks side by side as in a ring.  kExactRing, for
// calls that without rings would be walked: R~ and P_rb W~ each meet the state in a product (4.084e-3).  That product costs a block of a
// full device some 5 % (us, B=5, H=16, T=1000: 93.6 / 97.7; 40 heads, T=1999: 83.8 / 90), so that rings in the place of blocks side by
// side leave it out.
enum Form { kWalkForm, kBlocksForm, kRingForm, kExactRingForm };
//
// 256 threads: warp = (quad, hsel); quad selects the 32 TMEM lanes (tile rows) the warp may access,
// hsel the column half it works on, so every accumulator tile is shared by two warps per row group.
template <Form kForm>
__global__ void __launch_bounds__(256, 2)
wkv7_chunk_fwd_kernel(int Tlen, int H, int n_seq, const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ r,
                      const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ v,
                      const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b,
                      const __nv_bfloat16* __restrict__ s0, const uint32_t* __restrict__ length,
                      const uint8_t* __restrict__ new_starts, __nv_bfloat16* __restrict__ y,
                      __nv_bfloat16* __restrict__ s_out, float* __restrict__ s_at_len,
                      const __grid_constant__ StreamMaps maps, const __grid_constant__ CUtensorMap y_map, const __grid_constant__ CUtensorMap rbar_map,
                      unsigned char* __restrict__ saved,
                      int* __restrict__ range_flag, int range_ticket, int* __restrict__ residual_mark,
                      __nv_bfloat16* __restrict__ mprime, __nv_bfloat16* __restrict__ rbar, float* __restrict__ lam_out, int pieces,
                      const BlockParts parts) {
    constexpr bool kBlocks = kForm == kBlocksForm, kExactRing = kForm == kExactRingForm, kRing = kForm == kRingForm || kExactRing, kZero = kBlocks || kRing;
    if (kZero) let_next_in();
    extern __shared__ __align__(1024) unsigned char smem[];   // (the swizzle of the output tile is a function of the address)
    Small& sm = *reinterpret_cast<Small*>(smem + OFF_SMALL);
    // (all first pieces come first in the grid: where no cut exists the other pieces' CTAs return at once, and the
    // CTAs that do the work are then spread over the SMs before any SM takes a second one)
    const int nSlot = block_slots(Tlen);
    // blocks [unit, unit_end) of the list are this CTA's
    const int units = kBlocks ? n_seq * (nSlot - 1) : 0;
    int unit = kBlocks ? (int)((long long)units * blockIdx.x / gridDim.x) : 0;
    const int unit_end = kBlocks ? (int)((long long)units * (blockIdx.x + 1) / gridDim.x) : 0;
    const uint32_t ring_rank = kRing ? tc::cluster_rank() : 0, ring_size = kRing ? tc::cluster_size() : 1;
    int bh = kBlocks ? unit / (nSlot - 1) : kRing ? (int)(blockIdx.x / ring_size) : blockIdx.x % n_seq;
    const int piece = kZero ? 0 : blockIdx.x / n_seq;
    int bi = bh / H, h = bh % H;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int quad = warp & 3, hsel = warp >> 2;
    const int row = quad * 32 + lane;
    int L = min((int)length[bi], Tlen);
    // a ring's steps: the slots of the sequence in order of time, this CTA's are `step`, step + ring_size, ...
    const int bl = L / kC;
    const bool cut = kRing && slot_tokens(nSlot - 1, Tlen, L).n > 0;
    const int steps = cut ? nSlot : nSlot - 1;
    auto slot_of = [&](int m) { return !cut || m <= bl ? m : m == bl + 1 ? nSlot - 1 : m - 1; };
    int step = (int)ring_rank;
    // ---- sequence-parallel mode (pieces > 1, calls without a residual): a start flag cuts every dependence, so a
    // sequence may be walked as independent pieces whose first token carries a start flag.  Cut k, k = 1..pieces-1,
    // is the start flag nearest to k T / pieces within half a piece of it, if there is one; every CTA of the
    // sequence finds the same cuts by itself, a CTA whose own cut does not exist has nothing to do.
    int t_begin = 0, t_end = Tlen;
    if (kBlocks) t_begin = (unit - bh * (nSlot - 1)) * kC;
    if (kRing && step < steps) t_begin = slot_tokens(slot_of(step), Tlen, L).p;
    if (!kZero && pieces > 1) {
        const uint8_t* ns_row = new_starts + (size_t)bi * Tlen;
        const int half = Tlen / (2 * pieces);
        auto find_cut = [&](int k) -> int {       // position of cut k, or -1; all threads of the CTA take part
            const int target = (int)((long long)k * Tlen / pieces);
            const int lo = max(target - half, 1), hi = min(target + half, Tlen);
            __syncthreads();
            if (tid == 0) sm.nsm[0] = 0xffffffffu;
            __syncthreads();
            for (int t = lo + tid; t < hi; t += blockDim.x)
                if (ns_row[t] != 0) atomicMin(&sm.nsm[0], (uint32_t)(abs(t - target) * 2 + (t > target ? 1 : 0)) << 16 | (uint32_t)(t - lo));
            __syncthreads();
            const uint32_t best = sm.nsm[0];
            return best == 0xffffffffu ? -1 : lo + (int)(best & 0xffffu);
        };
        if (piece > 0) {
            t_begin = find_cut(piece);
            if (t_begin < 0) return;              // (the decision is the same for every thread)
        }
        for (int k = piece + 1; k < pieces; ++k) {
            const int c = find_cut(k);
            if (c >= 0) { t_end = c; break; }
        }
        __syncthreads();
    }
    const size_t tok_stride = (size_t)H * kN;
    size_t seq_base = (size_t)bi * Tlen * tok_stride + (size_t)h * kN;
    const size_t st_row = ((size_t)bh * kN + (row & 63)) * kN + hsel * 32;  // this thread's 32 state elements

    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < 5; ++i) tc::mbar_init(&sm.bar[i], (i == 2 || i == 3) ? 2 : 1);   // M3, M4: two issuing threads
        if (kRing) {
            tc::mbar_init(&sm.ring[0], 1);
            tc::mbar_init(&sm.ring[1], 1);
            tc::mbar_init(&sm.ring[2], 1);
            tc::mbar_init(&sm.ring[3], 1);
        }
        tc::mbar_init_fence();
        if (blockIdx.x == 0 && residual_mark != nullptr) *residual_mark = 0;   // this residual is in the chunked format (so far)
    }
    if (warp == 0) tc::tmem_alloc(&sm.tmem, 256);
    tc::fence_before_sync();
    if (kRing) tc::cluster_sync(); else __syncthreads();   // (the barriers of every CTA of the ring are there)
    tc::fence_after_sync();
    const uint32_t tbase = sm.tmem;
    const uint32_t lane_addr = tbase + ((uint32_t)(quad * 32) << 16);  // this warp's 32 TMEM lanes
    const uint32_t D1 = 0, D2 = 128, DS = 192;                        // TMEM column offsets (D3 aliases D1)
    bool failed = false;

    // ---- state into TMEM (rows 0..63 = S0 in fp32, rows 64..127 are never read) --------------
    if (!kZero) {
        float s[32];
        if (row < 64 && t_begin == 0) {
#pragma unroll
            for (int c = 0; c < 4; ++c) unpack8(*reinterpret_cast<const uint4*>(s0 + st_row + c * 8), &s[c * 8]);
        } else {
#pragma unroll
            for (int c = 0; c < 32; ++c) s[c] = 0.f;
        }
        tc::tmem_st32(lane_addr + DS + hsel * 32, s);
        tc::tmem_wait_st();
    }

    const uint32_t sAR = tc::smem_u32(smem + OFF_AR), sBK = tc::smem_u32(smem + OFF_BK);
    const uint32_t sBH = tc::smem_u32(smem + OFF_BH), sKH = tc::smem_u32(smem + OFF_KH);
    const uint32_t sSA = tc::smem_u32(smem + OFF_SA), sV = tc::smem_u32(smem + OFF_V);
    const uint32_t sM2A = tc::smem_u32(smem + OFF_M2A), sG = tc::smem_u32(smem + OFF_G);
    const uint32_t sTP = tc::smem_u32(smem + OFF_TP), sS0 = tc::smem_u32(smem + OFF_S0);
    constexpr uint32_t ID_128x128_KK = tc::make_idesc(128, 128, false, false);
    constexpr uint32_t ID_128x64_KK = tc::make_idesc(128, 64, false, false);
    constexpr uint32_t ID_128x64_KM = tc::make_idesc(128, 64, false, true);
    constexpr uint32_t ID_128x64_MM = tc::make_idesc(128, 64, true, true);

    float* cum = reinterpret_cast<float*>(smem + OFF_CUM);  // [64][LF_PITCH]
    float* lf = reinterpret_cast<float*>(smem + OFF_LF);    // [64][LF_PITCH]
    float* xinv = reinterpret_cast<float*>(smem + OFF_X);   // [64][LF_PITCH]
    float* scr = reinterpret_cast<float*>(smem + OFF_SCR);
    const int tsub = tid >> 3, jb = tid & 7;                // staging unit: tokens 32q+tsub (q=0,1), channels 8jb..8jb+7

    constexpr int kIssuer2 = 96;   // a thread of the warp with the least epilogue work
    int p = t_begin;
    uint32_t par = 0, spar = 0;   // phase parities of the product barriers and of the staging barrier
    // result tiles of the chunk just finished, waiting in shared memory for the next CTA barrier
    bool pend_y = false, pend_m = false, pend_r = false;
    int pend_p = 0;
    size_t pend_slot = 0;
    auto send_tiles = [&]() {   // behind a CTA barrier that follows the epilogue's stores
        if (warp == 7 && lane == 0 && (pend_y || pend_m)) {
            if (pend_y) tc::tensor_store_2d(&y_map, h * kN, bi * Tlen + pend_p, smem + OFF_YT);
            if (pend_m) {
                tc::bulk_store(mprime + pend_slot * (kN * kN), smem + OFF_MT, GTILE);
                // R- = R~ + P_rb W~: added in bf16 onto the R~ rows that went to global memory when the operands were scaled
                if (pend_r) tc::tensor_reduce_add_2d(&rbar_map, h * kN, bi * Tlen + pend_p, smem + OFF_RT);
            }
            tc::bulk_commit();
        }
        pend_y = pend_m = pend_r = false;
    };
    uint32_t in_par = 0, ready_par = 0, ring_par = 0;     // of the entering states, the next CTA's readiness, the state products
    if (kRing && L == 0 && step == 0 && quad < 2) {      // the input state comes back as it was given
        float s[32];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const uint4 raw = *reinterpret_cast<const uint4*>(s0 + st_row + c * 8);
            *reinterpret_cast<uint4*>(s_out + st_row + c * 8) = raw;
            unpack8(raw, &s[c * 8]);
        }
        if (s_at_len != nullptr) {
#pragma unroll
            for (int c = 0; c < 8; ++c)
                *reinterpret_cast<float4*>(s_at_len + st_row + c * 4) = make_float4(s[c * 4], s[c * 4 + 1], s[c * 4 + 2], s[c * 4 + 3]);
        }
    }
    uint8_t flag_ahead = (tid < 64 && t_begin + tid < Tlen) ? new_starts[(size_t)bi * Tlen + t_begin + tid] : 0;
    // the 64 token rows from cp on of w, r, k, v, a, b into the staging tiles (thread 0; one tiled copy
    // per stream).  Rows past the chunk arrive too and are ignored.
    auto issue_stage = [&](int cbi, int ch, int cp) {
        if (tid == 0) {
            tc::mbar_expect_tx(&sm.bar[4], (uint32_t)(6 * STG_TILE));
#pragma unroll
            for (int m = 0; m < 6; ++m) tc::tensor_load_2d(smem + stage_off(m), &maps.m[m], ch * kN, cbi * Tlen + cp, &sm.bar[4]);
        }
    };
    if (!kRing || step < steps) issue_stage(bi, h, t_begin);
    while (true) {
        // ================= boundary at position p: TMEM holds the state after token p-1 =================
        // (of the pieces of a sequence, the one that has walked token L - 1 holds it; L == 0: the first)
        const bool want_out = !kZero && (p == L) && (p > t_begin || t_begin == 0);
        if (quad < 2 && want_out) {
            float s[32];
            tc::tmem_ld32(lane_addr + DS + hsel * 32, s);
            tc::tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < 4; ++c) *reinterpret_cast<uint4*>(s_out + st_row + c * 8) = pack8(&s[c * 8]);
            if (s_at_len != nullptr) {
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    *reinterpret_cast<float4*>(s_at_len + st_row + c * 4) = make_float4(s[c * 4], s[c * 4 + 1], s[c * 4 + 2], s[c * 4 + 3]);
            }
        }
        if (kBlocks ? unit >= unit_end : kRing ? step >= steps : p >= t_end) break;
        // ================= extent of this chunk =================
        // (with a residual the chunks are the 64-token blocks of the sequence, so that the backward can number them)
        const int be = min(kBlocks || saved != nullptr ? ((p >> 6) + 1) << 6 : p + kC, t_end);
        const int p1 = kRing ? p + slot_tokens(slot_of(step), Tlen, L).n : L > p && L < be ? L : be, n = p1 - p;
        // what is walked next: the second part of this block, the next block, or the first of the next sequence; a ring's next step
        const bool next_seq = kBlocks && p1 == Tlen;
        const bool more = kBlocks ? p1 < be || unit + 1 < unit_end : kRing ? step + (int)ring_size < steps : p1 < t_end;
        const int np = kRing ? slot_tokens(slot_of(more ? step + (int)ring_size : step), Tlen, L).p : next_seq ? 0 : p1, nh = next_seq ? (h + 1 == H ? 0 : h + 1) : h, nbi = next_seq && h + 1 == H ? bi + 1 : bi;
        if (tid < 64) {
            // the flag byte of position p + tid was requested while the previous chunk's products ran
            const bool f = tid < n && flag_ahead != 0;
            const uint32_t m = __ballot_sync(0xffffffffu, f);
            if (lane == 0) sm.nsm[warp] = m;
        }
        __syncthreads();   // nsm visible; previous chunk's shared-memory readers are done
        send_tiles();
        const uint64_t mask = (uint64_t)sm.nsm[0] | ((uint64_t)sm.nsm[1] << 32);
        const bool reset_here = (mask & 1ull) != 0, inner = (mask >> 1) != 0, flagged = mask != 0;   // a flag on the first token; on others
        // the chunk leaves its operand slabs T, A_ak, P_rb, P_rk, sa, S0 for the backward: slot p / 64, and the last slot for
        // the second part of a block that `length` cuts (the only chunk that starts inside a block)
        const size_t blk_slot = (size_t)bh * nSlot + ((p & (kC - 1)) == 0 ? p >> 6 : nSlot - 1);
        unsigned char* const keep = saved != nullptr ? saved + blk_slot * kSavedBytes : nullptr;
        const bool affine = kZero || keep != nullptr;   // M', R- and L_C are wanted
        // ================= stage inputs (registers), log-decay into the scan buffer =================
        uint4 raw[2][5];   // r, k, v, a, b
        float lw[2][8];    // log2 of the decay: -exp(w) * log2(e)
        if (!tc::mbar_wait(&sm.bar[4], spar)) failed = true;   // the rows of this chunk have landed
        spar ^= 1u;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int t = q * 32 + tsub;
            if (t < n) {
                const int o = t * (kN * 2) + jb * 16;
                float wf[8];
                unpack8(*reinterpret_cast<const uint4*>(smem + stage_off(0) + o), wf);
#pragma unroll
                for (int m = 0; m < 5; ++m) raw[q][m] = *reinterpret_cast<const uint4*>(smem + stage_off(m + 1) + o);
#pragma unroll
                for (int e = 0; e < 8; ++e) lw[q][e] = -kLog2e * __expf(wf[e]);   // log2 of the decay
            } else {
#pragma unroll
                for (int m = 0; m < 5; ++m) raw[q][m] = make_uint4(0, 0, 0, 0);
#pragma unroll
                for (int e = 0; e < 8; ++e) lw[q][e] = 0.f;
            }
            // (column 4 jb + e holds channel 8 jb + e, column 32 + 4 jb + e channel 8 jb + 4 + e: the eight lanes of a
            // token then write, and later read, 128 contiguous bytes)
            *reinterpret_cast<float4*>(&cum[t * LF_PITCH + jb * 4]) = make_float4(lw[q][0], lw[q][1], lw[q][2], lw[q][3]);
            *reinterpret_cast<float4*>(&cum[t * LF_PITCH + 32 + jb * 4]) = make_float4(lw[q][4], lw[q][5], lw[q][6], lw[q][7]);
        }
        __syncthreads();
        if (tid < 128) {   // inclusive scan over tokens, two independent halves of 32 per channel
            const int j = tid & 63, half = tid >> 6;
            float run = 0.f;
#pragma unroll 8
            for (int tt = 0; tt < 32; ++tt) {
                const int t = half * 32 + tt;
                run += cum[t * LF_PITCH + j];
                cum[t * LF_PITCH + j] = run;
            }
            // column j of the scan buffer is channel ch = 8 jb + e
            const int cjb = (j & 31) >> 2, ce = (j & 3) + ((j >> 5) << 2), ch = cjb * 8 + ce;
            if (half == 0) sm.h1[ce * 8 + cjb] = run;
            else sm.tot[ch] = run;   // second-half sum for now
        }
        __syncthreads();
        if (tid < 64) {
            const float total = sm.h1[(tid & 7) * 8 + (tid >> 3)] + sm.tot[tid];
            // A decay so strong that 1 / L leaves the range the products can carry (never reached by decays
            // of the model's own parametrisation): the chunked form cannot represent this chunk.  Record it;
            // the token-sequential kernel launched behind this one redoes the call when it finds the mark.
            if (!(total >= kCumFloor)) atomicExch(range_flag, range_ticket);   // (or is no number)
            const float t2 = fmaxf(total, kCumFloor);
            sm.tot[tid] = t2;
            const float lam_c = ex2(t2);
            sm.lam[tid] = lam_c;
            sm.lamt[(tid & 7) * 8 + (tid >> 3)] = lam_c;
        }
        if (warp == 7) tc::bulk_wait_read<0>();   // the result tiles have left the slabs that are written next
        __syncthreads();
        // ================= scaled operands into the slabs =================
        {
            float h1v[8], lamv[8];   // first-half totals; 2^(chunk total) per channel
#pragma unroll
            for (int e = 0; e < 8; ++e) { h1v[e] = sm.h1[e * 8 + jb]; lamv[e] = sm.lamt[e * 8 + jb]; }
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int t = q * 32 + tsub;
                float c[8];
                *reinterpret_cast<float4*>(&c[0]) = *reinterpret_cast<const float4*>(&cum[t * LF_PITCH + jb * 4]);
                *reinterpret_cast<float4*>(&c[4]) = *reinterpret_cast<const float4*>(&cum[t * LF_PITCH + 32 + jb * 4]);
                float eL[8], eI[8], eP[8], eE[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float cc = fmaxf(c[e] + (q == 1 ? h1v[e] : 0.f), kCumFloor);
                    const float cp = fminf(fmaxf(cc - lw[q][e], kCumFloor), 0.f);   // cumulative log2-decay before this token
                    eL[e] = ex2(cc); eI[e] = ex2(-cc); eP[e] = ex2(cp);
                    eE[e] = lamv[e] * eI[e];   // 2^(total - cc) without a fourth trip to the special-function unit
                }
                // raw: r, k, v, a, b
                const uint4 a_t = scale8(raw[q][3], eP), r_t = scale8(raw[q][0], eL);
                slab_store(smem + OFF_AR, CB128, t, jb, a_t);
                slab_store(smem + OFF_AR, CB128, 64 + t, jb, r_t);
                if (affine) {
                    // W~ = T A~ is formed after the inverse, when the [A~ ; R~] slab has long been written over:
                    // a second copy of A~ waits in the sa slab, which is idle until sa itself is stored; R~ goes
                    // to the R- rows in global memory, where P_rb W~ is added at the end of the chunk
                    slab_store(smem + OFF_SA, CB64, t, jb, a_t);
                    if (t < n) *reinterpret_cast<uint4*>(rbar + seq_base + (size_t)(p + t) * tok_stride + jb * 8) = r_t;
                    tc::fence_async_global();   // a bulk copy adds onto these rows at the end of the chunk
                }
                slab_store(smem + OFF_BK, CB128, t, jb, scale8(raw[q][4], eI));
                slab_store(smem + OFF_BK, CB128, 64 + t, jb, scale8(raw[q][1], eI));
                slab_store(smem + OFF_BH, CB64, t, jb, scale8(raw[q][4], eE));
                slab_store(smem + OFF_KH, CB64, t, jb, scale8(raw[q][1], eE));
                slab_store(smem + OFF_V, CB64, t, jb, raw[q][2]);
            }
            if (flagged) {   // the rare chunk with start flags: the masked rows are written over
                const uint64_t m = start_mask(sm);
                __nv_bfloat162 odd = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int t = q * 32 + tsub;
#pragma unroll
                    for (int i = 1; i < 5; ++i)
                        if (!kZero) add_odd(odd, raw[q][i]);
                    const uint4 none = make_uint4(0, 0, 0, 0);
                    if (affine && !in_first(m, t)) {   // what carries the dependence on S0: nothing from the first flag on
                        slab_store(smem + OFF_SA, CB64, t, jb, none);
                        if (t < n) *reinterpret_cast<uint4*>(rbar + seq_base + (size_t)(p + t) * tok_stride + jb * 8) = none;
                        tc::fence_async_global();
                    }
                    if (!in_last(m, t)) {                       // what reaches S_C: nothing in front of the last flag
                        slab_store(smem + OFF_BH, CB64, t, jb, none);
                        slab_store(smem + OFF_KH, CB64, t, jb, none);
                    }
                }
                if (!kZero && is_odd(odd)) atomicExch(range_flag, range_ticket);
            }
        }
        // ================= entering state: bf16 copy for the products, decayed fp32 copy back to TMEM =====
        if (!kZero && quad < 2) {
            float s[32];
            if (reset_here) {
#pragma unroll
                for (int c = 0; c < 32; ++c) s[c] = 0.f;
            } else {
                tc::tmem_ld32(lane_addr + DS + hsel * 32, s);
                tc::tmem_wait_ld();
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) slab_store(smem + OFF_S0, CB64, row, hsel * 4 + c, pack8(&s[c * 8]));
            if (flagged) {
                float odd = 0.f;
#pragma unroll
                for (int c = 0; c < 32; ++c) odd = fmaf(s[c], 0.f, odd);
                if (odd != 0.f) atomicExch(range_flag, range_ticket);
            }
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const float4 l4 = *reinterpret_cast<const float4*>(&sm.lam[hsel * 32 + c * 4]);
                s[c * 4] *= l4.x; s[c * 4 + 1] *= l4.y; s[c * 4 + 2] *= l4.z; s[c * 4 + 3] *= l4.w;
            }
            if (flagged) {
#pragma unroll
                for (int c = 0; c < 32; ++c) s[c] = 0.f;
            }
            tc::tmem_st32(lane_addr + DS + hsel * 32, s);
            tc::tmem_wait_st();
        }
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        // ================= M1: pairwise products and the S0 products =================
        if (tid == 0) {
            tc::fence_after_sync();
            mma_k64(tbase + D1, kmaj128(sAR), kmaj128(sBK), ID_128x128_KK, false);
            if (!kZero) mma_k64(tbase + D2, kmaj128(sAR), kmaj64(sS0), ID_128x64_KK, false);
            tc::commit(&sm.bar[0]);
        }
        if (!kZero && keep != nullptr && warp == 7 && lane < 8) {   // the bf16 entering state goes to the residual as it is
            tc::bulk_store(keep + (size_t)SAVED_S0 * GTILE + lane * GCB, smem + OFF_S0 + lane * CB64, 64 * 16);
            tc::bulk_commit();
        }
        if ((kRing ? keep != nullptr : affine) && tid < 64) lam_out[blk_slot * kN + tid] = flagged ? 0.f : sm.lam[tid];
        if (!tc::mbar_wait(&sm.bar[0], par)) failed = true;
        tc::fence_after_sync();
        // ================= E1: triangular masks, operands of the next products =================
        if (inner) mask_pairs(lane_addr + D1 + hsel * 64, start_mask(sm), row & 63);
        {
            const int t = row & 63;
            float d[64];
            tc::tmem_ld32(lane_addr + D1 + hsel * 64, d);
            tc::tmem_ld32(lane_addr + D1 + hsel * 64 + 32, d + 32);
            tc::tmem_wait_ld();
            if (row < 64 && hsel == 0) {          // A_ab, strictly lower, fp32 for the inverse
#pragma unroll
                for (int c = 0; c < 16; ++c)
                    *reinterpret_cast<float4*>(&lf[t * LF_PITCH + c * 4]) =
                        make_float4(c * 4 + 0 < t ? d[c * 4 + 0] : 0.f, c * 4 + 1 < t ? d[c * 4 + 1] : 0.f,
                                    c * 4 + 2 < t ? d[c * 4 + 2] : 0.f, c * 4 + 3 < t ? d[c * 4 + 3] : 0.f);
            } else {
                const int lim = (row < 64) ? t : t + 1;   // A_ak strict; P_rb, P_rk inclusive
#pragma unroll
                for (int s = 0; s < 64; ++s) d[s] = (s < lim) ? d[s] : 0.f;
                // A_ak -> M2A rows 0..63, P_rk -> M2A rows 64..127, P_rb -> TP rows 64..127
                unsigned char* dst = smem + ((hsel == 1) ? OFF_M2A : OFF_TP);
#pragma unroll
                for (int c = 0; c < 8; ++c) slab_store(dst, CB128, row, c, pack8(&d[c * 8]));
            }
        }
        if (!kZero && inner) mask_state_products(lane_addr + D2 + hsel * 32, start_mask(sm), row & 63);
        if (warp == 7) tc::bulk_wait_read<0>();   // the S0 slab has been read: the inverse writes over part of it next
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        // ================= M2: G += A_ak V, Ypart += P_rk V ; meanwhile the triangular inverse =================
        if (tid == 0) {
            tc::fence_after_sync();
            mma_k64(tbase + D2, kmaj128(sM2A), mnmaj64(sV), ID_128x64_KM, !kZero);
            tc::commit(&sm.bar[1]);
        }
        // A_ak, P_rk and P_rb leave for the residual as bulk copies out of their slabs (one 64-row column
        // block of 1 KB per lane of the last warp); the copies must have read M2A before G is written over it,
        // which the hook in front of the inverse's last barrier guarantees
        if (keep != nullptr && warp == 7 && lane < 24) {
            const int which = lane >> 3, c = lane & 7;   // 0: A_ak, 1: P_rk, 2: P_rb
            const unsigned char* src = smem + (which == 2 ? OFF_TP : OFF_M2A) + c * CB128 + (which == 0 ? 0 : 64 * 16);
            unsigned char* dst = keep + (size_t)(which == 0 ? SAVED_AAK : (which == 1 ? SAVED_PRK : SAVED_PRB)) * GTILE + c * GCB;
            tc::bulk_store(dst, src, 64 * 16);
            tc::bulk_commit();
        }
        tri_inverse_64<256>(lf, xinv, scr, tid, [&]() { if (warp == 7) tc::bulk_wait_read<0>(); });
        fp32_to_slab64<256>(xinv, smem + OFF_TP, CB128, tid);
        if (quad < 2) {
            if (!tc::mbar_wait(&sm.bar[1], par)) failed = true;
            tc::fence_after_sync();
            float g[32];
            tc::tmem_ld32(lane_addr + D2 + hsel * 32, g);
            tc::tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < 4; ++c) slab_store(smem + OFF_G, CB64, row, hsel * 4 + c, pack8(&g[c * 8]));
        }
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        if (keep != nullptr && warp == 7 && lane < 8) {   // T: rows 0..63 of the [Tinv ; P_rb] slab
            tc::bulk_store(keep + (size_t)SAVED_T * GTILE + lane * GCB, smem + OFF_TP + lane * CB128, 64 * 16);
            tc::bulk_commit();
        }
        // ================= M3: sa = Tinv G =================
        if (tid == 0) {
            tc::fence_after_sync();
            mma_k64(tbase + D1, kmaj128(sTP), mnmaj64(sG), ID_128x64_KM, false);
            tc::commit(&sm.bar[2]);
        } else if (tid == kIssuer2) {   // what only the backward's carry needs is issued by a second thread
            tc::fence_after_sync();
            if (affine) mma_k64(tbase + D1 + 64, kmaj128(sTP), mnmaj64(sSA), ID_128x64_KM, false);   // W~ = Tinv A~
            tc::commit(&sm.bar[2]);
        }
        // the rows of the next chunk start travelling: their tiles lie over buffers that are idle from
        // here to the next chunk's operand stores (the inverse and the A_ak / P_rk product are done)
        if (more) issue_stage(nbi, nh, np);
        const int nL = next_seq && more ? min((int)length[nbi], Tlen) : L;
        if (quad < 2) {
            if (!tc::mbar_wait(&sm.bar[2], par)) failed = true;
            tc::fence_after_sync();
            float sa[32];
            tc::tmem_ld32(lane_addr + D1 + hsel * 32, sa);
            tc::tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < 4; ++c) slab_store(smem + OFF_SA, CB64, row, hsel * 4 + c, pack8(&sa[c * 8]));
            if (kZero && keep != nullptr) store_part(parts.sa, blk_slot, hsel, row, sa);
            if (affine) {
                tc::tmem_ld32(lane_addr + D1 + 64 + hsel * 32, sa);
                tc::tmem_wait_ld();
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const uint4 w16 = pack8(&sa[c * 8]);
                    slab_store(smem + OFF_G, CB64, row, hsel * 4 + c, w16);
                    if (kBlocks && keep != nullptr) parts.w_tilde[blk_slot * 512 + (hsel * 4 + c) * 64 + row] = w16;
                }
            }
        }
        if (kRing && warp == 7) tc::bulk_wait_read<0>();   // (T has left its slab, which is written over behind the next products)
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        if (!kZero && keep != nullptr && warp == 7 && lane < 8) {   // sa
            tc::bulk_store(keep + (size_t)SAVED_SA * GTILE + lane * GCB, smem + OFF_SA + lane * CB64, 64 * 16);
            tc::bulk_commit();
        }
        // ================= M4: Y += P_rb sa ; S += sa^T B^ + V^T K^ =================
        if (tid == 0) {
            tc::fence_after_sync();
            mma_k64(tbase + D2, kmaj128(sTP), mnmaj64(sSA), ID_128x64_KM, true);
            mma_k64(tbase + DS, mnmaj64(sSA), mnmaj64(sBH), ID_128x64_MM, !kZero);
            mma_k64(tbase + DS, mnmaj64(sV), mnmaj64(sKH), ID_128x64_MM, true);
            tc::commit(&sm.bar[3]);
        } else if (tid == kIssuer2) {
            tc::fence_after_sync();
            if (affine) {
                // the transition's off-diagonal part M' = W~^T B^ (rows 0..63 of the accumulator are used) and
                // the state-dependent part of the outputs, P_rb W~ (rows 64..127)
                mma_k64(tbase + D1, mnmaj64(sG), mnmaj64(sBH), ID_128x64_MM, false);
                mma_k64(tbase + D1 + 64, kmaj128(sTP), mnmaj64(sG), ID_128x64_KM, false);
            }
            tc::commit(&sm.bar[3]);
        }
        if (tid < 64) flag_ahead = (more && np + tid < Tlen) ? new_starts[(size_t)nbi * Tlen + np + tid] : 0;   // next chunk's start flags
        if (kZero && flagged && quad < 2) {
            const int at = hsel * 4 * CB64 + row * 16;
            leave_to_sequential_if_odd(smem + OFF_SA + at, smem + OFF_G + at, smem + OFF_V + at, range_flag, range_ticket);
        }
        if (!tc::mbar_wait(&sm.bar[3], par)) failed = true;
        tc::fence_after_sync();
        if constexpr (kBlocks) {
            float x[32];
            if (quad < 2) {
                tc::tmem_ld32(lane_addr + DS + hsel * 32, x);
                tc::tmem_wait_ld();
                store_part(parts.state, blk_slot, hsel, row, x);
                tc::tmem_ld32(lane_addr + D1 + hsel * 32, x);          // M'[j][j'], row j = this thread's lane, as high + low parts
                tc::tmem_wait_ld();
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const uint4 high = pack8(&x[c * 8]);
                    float hf[8];
                    unpack8(high, hf);
#pragma unroll
                    for (int e = 0; e < 8; ++e) hf[e] = x[c * 8 + e] - hf[e];
                    const size_t at = blk_slot * 512 + (hsel * 4 + c) * 64 + row;
                    reinterpret_cast<uint4*>(mprime)[at] = high;
                    parts.m_low[at] = pack8(hf);
                }
            } else {
                const int t = row - 64;
                uint4* const to = reinterpret_cast<uint4*>(rbar + seq_base + (size_t)(p + min(t, n - 1)) * tok_stride + hsel * 32);
                uint4 rt[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) rt[c] = to[c];             // R~, stored when the operands were scaled
                tc::tmem_ld32(lane_addr + D2 + hsel * 32, x);
                tc::tmem_wait_ld();
                store_part(parts.out, blk_slot, hsel, t, x);
                tc::tmem_ld32(lane_addr + D1 + 64 + hsel * 32, x);
                tc::tmem_wait_ld();
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float rf[8];
                    unpack8(rt[c], rf);
#pragma unroll
                    for (int e = 0; e < 8; ++e) rf[e] += x[c * 8 + e];
                    if (t < n) to[c] = pack8(rf);
                }
            }
        } else if constexpr (kRing) {
            // (the slabs that the entering state is put over have been read)
            const uint32_t left = (ring_rank + ring_size - 1) % ring_size, right = (ring_rank + 1) % ring_size;
            if (tid == 0 && step > 0) {
                tc::mbar_expect_tx(&sm.ring[2], kN * kN * 4);
                tc::mbar_arrive_in_cta(tc::in_cta(&sm.ring[3], left));
            }
            float x[32];
            uint4 pw[4];                                               // P_rb W~ (kExactRing)
            if (quad < 2) {
                tc::tmem_ld32(lane_addr + D1 + hsel * 32, x);          // M'[j][j'], row j = this thread's lane, as high + low parts
                tc::tmem_wait_ld();
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const uint4 high = pack8(&x[c * 8]);
                    float hf[8];
                    unpack8(high, hf);
#pragma unroll
                    for (int e = 0; e < 8; ++e) hf[e] = x[c * 8 + e] - hf[e];
                    slab_store(smem + OFF_MH, CB64, row, hsel * 4 + c, high);
                    if (keep != nullptr) {
                        reinterpret_cast<uint4*>(mprime)[blk_slot * 512 + (hsel * 4 + c) * 64 + row] = high;
                        slab_store(smem + OFF_WR, CB128, row, hsel * 4 + c, *reinterpret_cast<const uint4*>(smem + OFF_G + (hsel * 4 + c) * CB64 + row * 16));
                    }
                    slab_store(smem + OFF_ML, CB64, row, hsel * 4 + c, pack8(hf));
                }
            } else {
                const int t = row - 64;
                uint4* const to = reinterpret_cast<uint4*>(rbar + seq_base + (size_t)(p + min(t, n - 1)) * tok_stride + hsel * 32);
                uint4 rt[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) rt[c] = to[c];             // R~, stored when the operands were scaled
                tc::tmem_ld32(lane_addr + D1 + 64 + hsel * 32, x);
                tc::tmem_wait_ld();
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float rf[8];
                    unpack8(rt[c], rf);
#pragma unroll
                    for (int e = 0; e < 8; ++e) rf[e] += x[c * 8 + e];
                    const uint4 r_bar = pack8(rf);
                    slab_store(smem + OFF_WR, CB128, row, hsel * 4 + c, kExactRing ? rt[c] : r_bar);
                    if (keep != nullptr && t < n) to[c] = r_bar;
                    if constexpr (kExactRing) {
                        pw[c] = pack8(&x[c * 8]);
                        if (keep == nullptr) slab_store(smem + OFF_WR, CB128, t, hsel * 4 + c, pw[c]);
                    }
                }
            }
            // ---- the leaving state: of a flagged block U, which waits for nothing, otherwise what becomes of the entering one
            auto pass_on = [&](const float* state) {
                if (step + 1 < steps) {
                    const uint32_t to = tc::in_cta(smem + OFF_IN, right), bar = tc::in_cta(&sm.ring[2], right);
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        tc::store_in_cta(to + (uint32_t)((hsel * 8 + c) * 64 + row) * 16, make_float4(state[c * 4], state[c * 4 + 1], state[c * 4 + 2], state[c * 4 + 3]), bar);
                }
                if (p1 == L) {                 // the returned state
#pragma unroll
                    for (int c = 0; c < 4; ++c) *reinterpret_cast<uint4*>(s_out + st_row + c * 8) = pack8(&state[c * 8]);
                    if (s_at_len != nullptr) {
#pragma unroll
                        for (int c = 0; c < 8; ++c)
                            *reinterpret_cast<float4*>(s_at_len + st_row + c * 4) = make_float4(state[c * 4], state[c * 4 + 1], state[c * 4 + 2], state[c * 4 + 3]);
                    }
                }
            };
            if (flagged && quad < 2) {
                if (step + 1 < steps && !tc::mbar_wait_cluster(&sm.ring[3], ready_par)) failed = true;
                tc::tmem_ld32(lane_addr + DS + hsel * 32, x);
                tc::tmem_wait_ld();
                pass_on(x);
            }
            // ---- the entering state
            float4* const entering = reinterpret_cast<float4*>(smem + OFF_IN);
            if (quad < 2) {
                if (step == 0) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) unpack8(*reinterpret_cast<const uint4*>(s0 + st_row + c * 8), &x[c * 8]);
                    store_part(entering, 0, hsel, row, x);
                } else {
                    if (!tc::mbar_wait_cluster(&sm.ring[2], in_par)) failed = true;
                    load_part(entering, 0, hsel, row, x);
                }
                if (flagged) {
                    float odd = 0.f;
#pragma unroll
                    for (int c = 0; c < 32; ++c) odd = fmaf(x[c], 0.f, odd);
                    if (odd != 0.f) atomicExch(range_flag, range_ticket);
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) slab_store(smem + OFF_SB, CB64, row, hsel * 4 + c, reset_here ? make_uint4(0, 0, 0, 0) : pack8(&x[c * 8]));
            }
            if (step > 0) in_par ^= 1u;
            tc::fence_async_smem();
            tc::fence_before_sync();
            __syncthreads();
            if (tid == 0 && !flagged) {
                tc::fence_after_sync();
                mma_k64(tbase + DS, kmaj64(tc::smem_u32(smem + OFF_SB)), mnmaj64(tc::smem_u32(smem + OFF_ML)), ID_128x64_KM, true);
                mma_k64(tbase + DS, kmaj64(tc::smem_u32(smem + OFF_SB)), mnmaj64(tc::smem_u32(smem + OFF_MH)), ID_128x64_KM, true);
                tc::commit(&sm.ring[0]);
            } else if (tid == kIssuer2) {      // what no other CTA waits for
                tc::fence_after_sync();
                const bool onto_y = kExactRing && keep == nullptr;     // (nobody wants W~ S0^T)
                mma_k64(tbase + (onto_y ? D2 : D1), kmaj128(tc::smem_u32(smem + OFF_WR)), kmaj64(tc::smem_u32(smem + OFF_SB)), ID_128x64_KK, onto_y);
                if (!kExactRing) tc::commit(&sm.ring[1]);
            }
            if (keep != nullptr && warp == 7 && lane < 8) {   // the bf16 entering state goes to the residual
                tc::bulk_store(keep + (size_t)SAVED_S0 * GTILE + lane * GCB, smem + OFF_SB + lane * CB64, 64 * 16);
                tc::bulk_commit();
            }
            // P_rb W~ behind the state products, as rows 64..127 of an operand that begins 64 rows in front of it (nobody reads the results of
            // rows 0..63).  With a residual W~ has the rows that it has without, and it goes where the low part of M' was read.
            if (kExactRing && quad >= 2) {
                if (!flagged && !tc::mbar_wait(&sm.ring[0], ring_par)) failed = true;
                if (keep != nullptr) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) slab_store(smem + OFF_PW, CB64, row - 64, hsel * 4 + c, pw[c]);
                    tc::fence_async_smem();
                    tc::fence_before_sync();
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                }
                if (tid == kIssuer2) {
                    tc::fence_after_sync();
                    mma_k64(tbase + D2, keep == nullptr ? kmaj128(tc::smem_u32(smem + OFF_WR) - 64 * 16) : kmaj64(tc::smem_u32(smem + OFF_PW) - 64 * 16),
                            kmaj64(tc::smem_u32(smem + OFF_SB)), ID_128x64_KK, true);
                    tc::commit(&sm.ring[1]);
                }
            }
            if (!flagged) {
                // (meanwhile: whether the next CTA can take the state, what remains of the entering one)
                if (quad < 2) {
                    if (step + 1 < steps && !tc::mbar_wait_cluster(&sm.ring[3], ready_par)) failed = true;
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const float4 l4 = *reinterpret_cast<const float4*>(&sm.lam[hsel * 32 + c * 4]);
                        x[c * 4] *= l4.x; x[c * 4 + 1] *= l4.y; x[c * 4 + 2] *= l4.z; x[c * 4 + 3] *= l4.w;
                    }
                }
                if (!tc::mbar_wait(&sm.ring[0], ring_par)) failed = true;
                ring_par ^= 1u;
                tc::fence_after_sync();
                if (quad < 2) {
                    float s[32];
                    tc::tmem_ld32(lane_addr + DS + hsel * 32, s);
                    tc::tmem_wait_ld();
#pragma unroll
                    for (int c = 0; c < 32; ++c) s[c] += x[c];
                    pass_on(s);
                }
            }
            if (step + 1 < steps) ready_par ^= 1u;
            // ---- outputs (and sa)
            if (!tc::mbar_wait(&sm.ring[1], par)) failed = true;
            tc::fence_after_sync();
            if (quad >= 2) {
                const int t = row - 64;
                float yv[32];
                tc::tmem_ld32(lane_addr + D2 + hsel * 32, yv);
                if (!kExactRing || keep != nullptr) {
                    tc::tmem_ld32(lane_addr + D1 + hsel * 32, x);
                    tc::tmem_wait_ld();
#pragma unroll
                    for (int c = 0; c < 32; ++c) yv[c] += x[c];
                } else {
                    tc::tmem_wait_ld();
                }
                if (n == kC) {
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        *reinterpret_cast<uint4*>(smem + OFF_YT + t * 128 + (((hsel * 4 + c) ^ (t & 7)) << 4)) = pack8(&yv[c * 8]);
                } else if (t < n) {
                    __nv_bfloat16* dst = y + seq_base + (size_t)(p + t) * tok_stride + hsel * 32;
#pragma unroll
                    for (int c = 0; c < 4; ++c) *reinterpret_cast<uint4*>(dst + c * 8) = pack8(&yv[c * 8]);
                }
            } else if (keep != nullptr) {
                float s[32];
                tc::tmem_ld32(lane_addr + D1 + hsel * 32, x);
                load_part(parts.sa, blk_slot, hsel, row, s);
                tc::tmem_wait_ld();
#pragma unroll
                for (int c = 0; c < 32; ++c) s[c] += x[c];
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    *reinterpret_cast<uint4*>(keep + (size_t)SAVED_SA * GTILE + (hsel * 4 + c) * GCB + row * 16) = pack8(&s[c * 8]);
            }
            pend_y = (n == kC);
            pend_p = p;
        } else {
        if (quad >= 2) {
            const int t = row - 64;
            float yv[32];
            tc::tmem_ld32(lane_addr + D2 + hsel * 32, yv);
            tc::tmem_wait_ld();
            if (n == kC) {        // a full block leaves as one tiled copy out of shared memory
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    *reinterpret_cast<uint4*>(smem + OFF_YT + t * 128 + (((hsel * 4 + c) ^ (t & 7)) << 4)) = pack8(&yv[c * 8]);
            } else if (t < n) {
                __nv_bfloat16* dst = y + seq_base + (size_t)(p + t) * tok_stride + hsel * 32;
#pragma unroll
                for (int c = 0; c < 4; ++c) *reinterpret_cast<uint4*>(dst + c * 8) = pack8(&yv[c * 8]);
            }
        }
        pend_y = (n == kC);
        pend_p = p;
        pend_m = (keep != nullptr);
        pend_r = pend_m && n == kC;
        pend_slot = blk_slot;
        if (keep != nullptr) {
            float m[32];
            if (quad < 2) {       // M'[j][j'], row j = this thread's lane
                tc::tmem_ld32(lane_addr + D1 + hsel * 32, m);
                tc::tmem_wait_ld();
#pragma unroll
                for (int c = 0; c < 4; ++c) slab_store(smem + OFF_MT, GCB, row, hsel * 4 + c, pack8(&m[c * 8]));
            } else {              // R-_t = R~_t + (P_rb W~)_t on top of the R~ row stored at the start of the chunk
                const int t = row - 64;
                if (n == kC) {
                    tc::tmem_ld32(lane_addr + D1 + 64 + hsel * 32, m);
                    tc::tmem_wait_ld();
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        *reinterpret_cast<uint4*>(smem + OFF_RT + t * 128 + (((hsel * 4 + c) ^ (t & 7)) << 4)) = pack8(&m[c * 8]);
                } else {              // a short chunk's rows one by one: a tiled copy would go over the next sequence's
                    add_to_row(lane_addr + D1 + 64 + hsel * 32, rbar + seq_base + (size_t)(p + t) * tok_stride + hsel * 32, t < n);
                }
            }
        }
        }
        tc::fence_async_smem();   // the result tiles are read by bulk copies
        tc::fence_before_sync();
        if (warp == 7) tc::bulk_wait_read<0>();   // the slabs copied out may be rewritten after the next barrier
        p = np;
        if (kRing) step += (int)ring_size;
        if (kBlocks) {
            if (p1 == be) ++unit;
            if (next_seq) {
                ++bh;
                bi = nbi;
                h = nh;
                L = nL;
                seq_base = (size_t)bi * Tlen * tok_stride + (size_t)h * kN;
            }
        }
        par ^= 1u;
    }
    __syncthreads();
    send_tiles();   // of the last chunk
    if (warp == 7) tc::bulk_wait_all<0>();   // every copy to the residual has landed before the CTA retires
    if (failed) atomicExch(&g_status, 1);
    tc::fence_before_sync();
    if (kRing) tc::cluster_sync(); else __syncthreads();   // (no CTA of a ring leaves while another one may still write to it)
    if (warp == 0) tc::tmem_dealloc(tbase, 256);
}

}  // namespace

size_t wkv7_chunk_residual_bytes(int B, int T, int H) { return residual_layout(B, T, H).end; }

// A forward call that meets a decay outside the chunked kernels' range tells the fallback launched behind
// it through one int of device memory.  Calls may be in flight on several streams, so each call takes the
// next slot of a small ring and a ticket that no earlier call used: a slot never needs clearing.
__device__ int g_range_flags[64];

static int* range_flag_ring() {
    static DeviceOnce once;
    static int* addr[kMaxDevices];
    const int dev = current_device();
    if (dev < 0) return nullptr;
    if (!once.ok([dev]() {
            int* ptr = nullptr;
            const cudaError_t e = cudaGetSymbolAddress((void**)&ptr, g_range_flags);
            addr[dev] = (e == cudaSuccess) ? ptr : nullptr;
            return e;
        }))
        return nullptr;
    return addr[dev];
}

// A slot of the ring and a ticket no earlier call used (never 0, so untouched memory cannot match); NULL on failure.
int* wkv_call_flag(int* ticket) {
    static std::atomic<unsigned> tickets{1};
    int* ring = range_flag_ring();
    if (ring == nullptr) return nullptr;
    const unsigned t = tickets.fetch_add(1);
    *ticket = (int)(t | 0x40000000u);
    return ring + (t & 63u);
}

// The rule between the three forms, as the bytes of workspace that rings and blocks side by side want (0: the sequential walk).
// Walking a sequence takes 6.6 us per block whatever else runs, up to one sequence per SM; side by side, a block costs 0.04 us
// of the device and a step of the chain 1.2-1.5 us, and two more launches and the workspace some 10 us of host time.  Measured
// (us, walk / side by side, forward of BH sequences without start flags): T=256: 37 / 36 at BH=40, 39 / 48 at 96; T=1024:
// 118 / 75 at 40, 119 / 92 at 64, 123 / 116 at 96; T=4096: 435 / 208 at 40, 437 / 265 at 64.  So: from four blocks on, up to
// half a sequence per SM.  With a residual up to two thirds of one in long sequences (BH=96: 243 / 227 at T=2048, 464 / 409
// at 4096).  Without one, the walk is cut at start flags where there are any, and then wins where there are many blocks
// (a flag every 256 tokens: 156 / 138 at BH=64, T=2048; 163 / 164 at 40, 181 / 227 at 64, T=4096): up to nine blocks per CTA
// slot.  The last limit bounds the workspace, 2 GiB.
//
// Rings take precedence.  A ring has as many CTAs as the device has room for: seven eighths of the two slots per SM, because a
// cluster stays within a GPC (BH=32, T=2048: 83 us by six, 72 by seven, 68 by eight; 114 by nine, which do not fit at once; two
// CTAs only wait for one another).  Nine are enough to keep a state moving (17 k cycles for a block, 2.7 k for a hop); up to a
// sixteenth of a sequence per SM there is room for sixteen, which halves the time between start flags.  Of four and more, a ring
// is the fastest without flags; a ring of three is slower than blocks side by side (which go up to half a sequence per SM) from eight
// blocks on.  With flags, blocks side by side and the walk in pieces are cut into shorter chains, a ring isn't, and loses in long
// sequences.  With a residual the walk is not cut, and a ring lasts longer.  The host doesn't know the flags: a limit in blocks lies where a
// ring and what is taken behind it are equal at a flag every 256 tokens, or where it loses 2-9 % with those and gains 7-24 % without
// (rings of four and six).  us, that form / ring (kRing; where that form is the walk the call takes kExactRing, 4 % above the figure
// here), without flags and with (rings of seven and more are the faster ones up to T=4096
// except of few heads, which don't fill the device):
//     no residual  BH=4, 8:   T=1536 52 / 46, 36 / 31 and 54 / 51, 43 / 39      2000 60 / 56, 34 / 36 and 64 / 62, 44 / 45     4096 112 / 108, 58 / 73
//                  BH=16:     T=1536 66 / 52, 54 / 50    1792 73 / 59, 55 / 55    4096 136 / 111, 89 / 104
//                  BH=24, 36: T=3072 125 / 92, 83 / 85 and 154 / 102, 119 / 108    4096 163 / 118, 112 / 112 and 196 / 132, 149 / 135
//                  BH=40:     T=2304 126 / 94, 100 / 95    2560 137 / 103, 108 / 109    3072 158 / 120, 121 / 125
//                  BH=48:     T=2304 139 / 113, 117 / 117    2560 150 / 124, 129 / 128    3072 178 / 143, 145 / 150
//                  BH=64:     T=1472 110 / 95, 104 / 100    1600 120 / 102, 111 / 106    1792 132 / 114, 118 / 118    2000 145 / 126, 126 / 133
//                  BH=56:     T=1600 112 / 100, 102 / 102    1792 122 / 113, 111 / 115    2000 136 / 127, 120 / 131
//                  BH=65-74:  T=192 25 / 22, 27 / 22    384 46 / 40, 46 / 42    448 50 / 44, 49 / 45    512 51 / 51, 50 / 53    1024 87 / 93, 82 / 96
//                  BH=80:     T=768 85 / 72, 76 / 74    1024 112 / 95, 102 / 95 (walked)    1280 138 / 114, 117 / 117    1536 165 / 133, 104 / 136
//     residual     BH=40, 48, 64: T=3072 177 / 136, 140 / 138 and 198 / 164, 167 / 167 and 232 / 207, 209 / 213      4096 224 / 174, 179 / 178 and
//                             251 / 206, 209 / 217 and 303 / 274, 265 / 279
//                  BH=65-74:  T=320 48 / 38, 50 / 38    384 52 / 46, 53 / 47    512 60 / 58, 59 / 60    1024 100 / 105, 95 / 107
//                  BH=80:     T=1024 121 / 105, 125 / 107 (walked)    1472 169 / 141, 174 / 145    1536 153 / 145, 141 / 149 (side by side from here on)
// From three blocks on (T=192: 25 / 19; two: 19 / 17-21), with a residual from four: there the host, who has a workspace to
// allocate, is what such a call waits for.
static int ring_size(long long sms, int largest, int B, int T, int H, bool residual) {
    const long long seqs = (long long)B * H, blocks = block_slots(T) - 1;
    const long long n = std::min(16 * seqs <= sms ? 16 : std::min(7 * sms / 4 / seqs, 9LL), (long long)largest);
    const bool few = 9 * seqs < 4 * sms / 3;                  // rings at their largest leave a third of the device idle
    const long long longest = few ? 24 : n >= 7 ? 65535 : n > 3 && residual ? 48 : n == 6 ? 48 : n == 5 ? 40 : n == 4 ? 32 : 2 * seqs <= sms ? 7 : residual ? 23 : 16;
    if (n < 3 || blocks < (residual ? 4 : 3) || blocks > longest) return 1;
    return (int)std::min(n, blocks);
}
// A ring's workspace.  With a residual: sa' of every slot, which waits there for the entering state.  Without: R~ of every token, which
// the residual would have room for.
static size_t ring_bytes(int B, int T, int H, bool residual) {
    return (size_t)B * H * (residual ? (size_t)block_slots(T) * (kC * kN * sizeof(float)) : (size_t)T * (kN * sizeof(__nv_bfloat16)));
}

// The form for a device of `sms` SMs that takes clusters of up to `largest` CTAs: the CTAs of a ring, or kWalkForm, kBlocksForm
constexpr size_t kMostWorkspace = (size_t)2 << 30;
static int form_without_rings(int sms, int B, int T, int H, bool residual) {
    const long long seqs = (long long)B * H, blocks = block_slots(T) - 1;
    if (blocks < 4 || blocks >= 65536) return kWalkForm;
    if (2 * seqs > sms && !(residual && blocks >= 24 && 3 * seqs <= 2 * sms)) return kWalkForm;
    if (!residual && seqs * blocks > 9LL * 2 * sms) return kWalkForm;
    return blocks_layout(B, T, H, residual).end <= kMostWorkspace ? kBlocksForm : kWalkForm;
}
int wkv7_fwd_form(int sms, int largest, int B, int T, int H, bool residual) {
    const int ring = ring_size(sms, largest, B, T, H, residual);
    return ring > 1 && ring_bytes(B, T, H, residual) <= kMostWorkspace ? ring : form_without_rings(sms, B, T, H, residual);
}

static cudaLaunchConfig_t ring_config(cudaLaunchAttribute* attr, int heads, int ring, cudaStream_t st) {
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = ring; attr->val.clusterDim.y = 1; attr->val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(heads * ring));
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}
static bool forms_set_up() {       // the opt-in to large dynamic shared memory is a per-device function attribute
    static DeviceOnce once;
    return once.ok([]() {
        cudaError_t e = cudaSuccess;
        for (const auto kernel : {wkv7_chunk_fwd_kernel<kWalkForm>, wkv7_chunk_fwd_kernel<kBlocksForm>, wkv7_chunk_fwd_kernel<kRingForm>, wkv7_chunk_fwd_kernel<kExactRingForm>})
            if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        for (const auto kernel : {wkv7_chunk_fwd_kernel<kRingForm>, wkv7_chunk_fwd_kernel<kExactRingForm>})
            if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        return e;
    });
}
// CTAs of the largest ring that the current device takes: 16 of a whole B200 (seven such clusters at once), fewer, down to none, where
// the process has been given a share of its SMs.
static int largest_ring() {
    static DeviceOnce once;
    static int largest[kMaxDevices];
    const int dev = current_device();
    if (dev < 0 || !forms_set_up()) return 0;
    once.ok([dev]() {
        for (int n = 16; n > 2 && largest[dev] == 0; --n) {
            cudaLaunchAttribute attr;
            const cudaLaunchConfig_t cfg = ring_config(&attr, 1, n, nullptr);
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, wkv7_chunk_fwd_kernel<kRingForm>, &cfg) != cudaSuccess) (void)cudaGetLastError();
            else if (clusters > 0) largest[dev] = n;
        }
        return cudaSuccess;
    });
    return largest[dev];
}
static int form_here(int B, int T, int H, bool residual) { return wkv7_fwd_form(sm_count_of_current_device(), largest_ring(), B, T, H, residual); }

size_t wkv7_blocks_bytes(int B, int T, int H, bool residual) {
    const int form = form_here(B, T, H, residual);
    return form == kWalkForm ? 0 : form == kBlocksForm ? blocks_layout(B, T, H, residual).end : ring_bytes(B, T, H, residual);
}

int wkv7_chunk_fwd(cudaStream_t st, int B, int T, int H, const void* w, const void* r, const void* k, const void* v,
                   const void* a, const void* b, const void* s0, const uint32_t* length, const uint8_t* ns, void* y,
                   void* s_out, void* residual, void* workspace, int* residual_mark, int** range_flag, int* range_ticket) {
    typedef __nv_bfloat16 bf;
    if (!forms_set_up()) return B200WKV_ELAUNCH;
    *range_flag = wkv_call_flag(range_ticket);
    if (*range_flag == nullptr) return B200WKV_ELAUNCH;
    const ResidualLayout lay = residual_layout(B, T, H);
    char* const base = static_cast<char*>(residual);
    StreamMaps maps;
    const void* bases[6] = {w, r, k, v, a, b};   // maps[m]: the six streams as [B*T tokens][H*64 channels]
    if (!make_stream_maps(&maps, bases, 6, B, T, H)) return B200WKV_ELAUNCH;
    StreamMaps out_maps;                         // m[0]: the outputs, with the 128-byte swizzle of the kernel's output tile
    const void* out_bases[2] = {y, residual ? (const void*)((char*)residual + lay.rbar) : y};   // m[1]: the R- rows
    if (!make_stream_maps(&out_maps, out_bases, 2, B, T, H, /*swizzle128=*/true)) return B200WKV_ELAUNCH;
    const int form = workspace != nullptr ? form_here(B, T, H, residual != nullptr) : (int)kWalkForm;      // (the workspace has the form's bytes)
    if (form > kBlocksForm) {
        BlockParts parts = {};
        parts.sa = (float4*)workspace;
        cudaLaunchAttribute attr;
        const cudaLaunchConfig_t cfg = ring_config(&attr, B * H, form, st);
        const bool walked = form_without_rings(sm_count_of_current_device(), B, T, H, residual != nullptr) == kWalkForm;
        if (cudaLaunchKernelEx(&cfg, walked ? wkv7_chunk_fwd_kernel<kExactRingForm> : wkv7_chunk_fwd_kernel<kRingForm>, T, H, B * H, (const bf*)w, (const bf*)r, (const bf*)k, (const bf*)v, (const bf*)a,
                               (const bf*)b, (const bf*)s0, length, ns, (bf*)y, (bf*)s_out, residual ? (float*)(base + lay.s_at_len) : (float*)nullptr, maps,
                               out_maps.m[0], out_maps.m[1], residual ? (unsigned char*)(base + lay.saved) : (unsigned char*)nullptr, *range_flag,
                               *range_ticket, residual_mark, residual ? (bf*)(base + lay.mprime) : (bf*)nullptr,
                               residual ? (bf*)(base + lay.rbar) : (bf*)workspace,
                               residual ? (float*)(base + lay.lam) : (float*)nullptr, 1, parts) == cudaSuccess)
            return B200WKV_OK;
        (void)cudaGetLastError();  // (a share of SMs that this stream alone has: the walk below needs no cluster)
    }
    if (form == kBlocksForm) {     // the blocks side by side
        const BlocksLayout bl = blocks_layout(B, T, H, residual != nullptr);
        char* const ws = static_cast<char*>(workspace);
        BlocksCall c;
        c.parts = BlockParts{(float4*)(ws + bl.state), (float4*)(ws + bl.out), (float4*)(ws + bl.sa), (uint4*)(ws + bl.m_low), (uint4*)(ws + bl.w_tilde)};
        c.saved = residual ? (unsigned char*)(base + lay.saved) : nullptr;
        c.mprime = residual ? (bf*)(base + lay.mprime) : (bf*)(ws + bl.mprime);
        c.rbar = residual ? (bf*)(base + lay.rbar) : (bf*)(ws + bl.rbar);
        c.lam = residual ? (float*)(base + lay.lam) : (float*)(ws + bl.lam);
        c.s0_tiles = residual ? c.saved + (size_t)SAVED_S0 * GTILE : (unsigned char*)(ws + bl.s0);
        c.s0_stride = residual ? kSavedBytes : (size_t)GTILE;
        const long long units = (long long)B * H * (block_slots(T) - 1), slots = 2LL * sm_count_of_current_device();
        wkv7_chunk_fwd_kernel<kBlocksForm><<<(int)(units < slots ? units : slots), 256, SMEM_BYTES, st>>>(
            T, H, B * H, (const bf*)w, (const bf*)r, (const bf*)k, (const bf*)v, (const bf*)a, (const bf*)b, (const bf*)s0, length, ns, (bf*)y,
            (bf*)s_out, nullptr, maps, out_maps.m[0], out_maps.m[1], c.saved, *range_flag, *range_ticket, residual_mark, c.mprime, c.rbar, c.lam, 1,
            c.parts);
        if (cudaGetLastError() != cudaSuccess) return B200WKV_ELAUNCH;
        return wkv7_blocks_finish(st, B, T, H, length, ns, s0, *range_flag, *range_ticket, c, y, s_out, residual ? (float*)(base + lay.s_at_len) : nullptr);
    }
    // Without a residual (inference) and with fewer sequences than CTA slots, every sequence is offered to several
    // CTAs, which cut it at start flags where there are any (see the kernel): at most 8 pieces of at least 128 tokens.
    int pieces = 1;
    if (residual == nullptr) {
        const long long slots = 2LL * sm_count_of_current_device();
        const long long seqs = (long long)B * H;
        if (seqs < slots) pieces = (int)((2 * slots + seqs - 1) / seqs);
        if (pieces > 8) pieces = 8;
        if (pieces > T / 128) pieces = T / 128;
        if (pieces < 1 || T / pieces >= 32768) pieces = 1;
    }
    wkv7_chunk_fwd_kernel<kWalkForm><<<B * H * pieces, 256, SMEM_BYTES, st>>>(T, H, B * H, (const bf*)w, (const bf*)r, (const bf*)k, (const bf*)v,
                                                          (const bf*)a, (const bf*)b, (const bf*)s0, length, ns,
                                                          (bf*)y, (bf*)s_out, residual ? (float*)(base + lay.s_at_len) : nullptr,
                                                          maps, out_maps.m[0], out_maps.m[1],
                                                          residual ? (unsigned char*)(base + lay.saved) : nullptr,
                                                          *range_flag, *range_ticket, residual_mark,
                                                          residual ? (bf*)(base + lay.mprime) : nullptr,
                                                          residual ? (bf*)(base + lay.rbar) : nullptr,
                                                          residual ? (float*)(base + lay.lam) : nullptr, pieces, BlockParts{});
    return cudaGetLastError() == cudaSuccess ? B200WKV_OK : B200WKV_ELAUNCH;
}

// Device address of the status word on the current device (resolved once per device).
int* wkv7_chunk_status_word() {
    static DeviceOnce once;
    static int* addr[kMaxDevices];
    const int dev = current_device();
    if (dev < 0) return nullptr;
    if (!once.ok([dev]() {
            int* ptr = nullptr;
            const cudaError_t e = cudaGetSymbolAddress((void**)&ptr, g_status);
            addr[dev] = (e == cudaSuccess) ? ptr : nullptr;
            return e;
        }))
        return nullptr;
    return addr[dev];
}

// Reads and clears the device-side error word (synchronises the device; diagnostics only).
int wkv7_chunk_status() {
    int h = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&h, g_status, sizeof(int)) != cudaSuccess) return -1;
    cudaMemcpyToSymbol(g_status, &zero, sizeof(int));
    return h;
}

}  // namespace b200wkv
