// RWKV-5 / 5.2 / 6 WKV recurrence in chunks of 16 tokens on the tensor cores (bf16 I/O, fp32 state).
//
// State S[key i][value j];  y_t = r_t (S_{t-1} + diag(u) k_t^T v_t),  S_t = diag(d_t) S_{t-1} + k_t^T v_t  with the decay
// d_t = exp(lw_t) per key channel (lw_t = w_t for RWKV-6, log of the head's constant for RWKV-5 / 5.2).  With the
// inclusive cumulative log-decay c_t inside a chunk (c_{-1} = 0, c_m at the chunk's middle, c_C at its end):
//     R0_t = r_t exp(c_{t-1})            K^_s = k_s exp(c_C - c_s)
//     R~_t = r_t exp(c_{t-1} - c_m)      K~_s = k_s exp(c_m - c_s)         (referenced to the middle: |exponent| <= 8 tokens)
//     A_ts = R~_t . K~_s  (s < t),  A_tt = sum_i r u k
//     Y = R0 S0 + A V                    S_C = diag(exp(c_C)) S0 + K^^T V
// A start flag on token p cuts every dependence of tokens >= p on tokens < p and on S0: masks on A, on the rows
// of R0 and of K^, and on the carried state.  The state is held transposed, S^T[j][i], as mma.sync accumulator
// tiles (fp32, each of the four warps 16 value rows): a tile is already in the register layout of the next
// product's left operand, and the 16x16 score block A, computed by every warp for itself, is already in the
// layout of a right operand, so nothing but the scaled operands passes through shared memory.  The chunk is 16
// tokens because the per-channel decay is unbounded: referenced to the chunk's middle the scaling factors stay
// below exp(8 |lw|), which fp32 / bf16 hold for |lw| <= 10 per token (decay >= 4.5e-5); a chunk beyond that, or a
// decay above 1, makes the kernel leave its ticket in a flag and the token-sequential kernels (wkv6_seq.cu) redo the
// call.  A `length` inside a chunk splits that chunk in two parts that are walked like two chunks.  tcgen05 does not
// apply: its smallest tile is 64 tokens.
//
// Semantics: BaseRWKV.inner_loop of jaxrwkv, src/jaxrwkv/rwkv6.py:174-191, rwkv5_2.py:164-180, rwkv5.py:161-177.
#include <type_traits>

#include "common.cuh"
#include "device_once.cuh"
#include "tc05.cuh"
#include "tmap.cuh"

namespace b200wkv {

int* wkv7_chunk_status_word();      // wkv7_chunk.cu: where a kernel leaves the code of a bounded wait that ran out
int* wkv_call_flag(int* ticket);   // wkv7_chunk.cu: a slot of the per-device flag ring and a fresh ticket

namespace {

typedef __nv_bfloat16 bf;
using tc::ldmatrix_x4;
using tc::ldmatrix_x4_trans;
using tc::mma_bf16;
constexpr int kC6 = 16;          // tokens per chunk
constexpr int kRunLen6 = 16;    // chunks per run of the run-parallel backward
constexpr int PITCH = 72;        // bf16 per shared-memory row (144 bytes): 4-byte fragment reads and ldmatrix rows hit 32 banks
constexpr float kMaxHalfDecay = 80.f;   // |sum of lw over half a chunk| the scaling can represent

// One 16-token x 16-channel block of a row-major [token][channel] tile, f[0..3] = (tokens 0-7 | 8-15) x (channels 0-7 |
// 8-15) in the order (0-7, 0-7), (8-15, 0-7), (0-7, 8-15), (8-15, 8-15).  As a LEFT operand (rows = tokens) the four
// are a0..a3; as a RIGHT operand (n = token, k = channel) tokens 0-7 take (f[0], f[2]) and tokens 8-15 (f[1], f[3]).
struct Frag {
    uint32_t f[4];
};
__device__ __forceinline__ void mma_ab(float* d, const Frag& a, const Frag& b, int nt) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a.f[0]), "r"(a.f[1]), "r"(a.f[2]), "r"(a.f[3]), "r"(b.f[nt]), "r"(b.f[nt + 2]));
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// exp in two instructions (results below the smallest normal number are zero; __expf spends three more on them)
__device__ __forceinline__ float exp_fast(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * 1.4426950408889634f));
    return y;
}

// ------------------------------------------------------------------ forward ---------
// What bounds it is the instructions of the operands' preparation (512 sequences of 256 chunks on 592 CTA slots: every
// chunk's instructions lie in one chain per CTA, four CTAs deep on an SM).  So a warp prepares the 16 channels that it also
// owns as value columns, for all 16 tokens, in the layout of the tensor cores' tiles: the cumulative log-decay, referenced to
// the chunk's middle, is a product of constant triangles of -1, 0, 1 with the raw log-decay rows (exact products, fp32 sums),
// so that it needs neither a scan nor another warp; its result lies where r and k of the same (token, channel) pairs can be
// read as words; and what leaves for shared memory are whole fragments (stmatrix).  One barrier per chunk.
// At B=16, T=4096, H=32: 0.55 ms with the residual (0.81 ms with the sums a scan over quarters of the
// chunk, 4-byte operand stores, and raw rows fetched by every thread).
constexpr int kRing6 = 3;        // raw rows of r, k, w: read before a chunk's barrier only
constexpr int kRingV6 = 4;       // raw rows of v: read behind it
constexpr int kTile6 = kC6 * kN * 2;     // bytes of a chunk's rows of one stream, as the tiled copies move them (rows of 128 bytes, swizzled)
struct Fwd6cSmem {
    unsigned char r[kRing6][kTile6], k[kRing6][kTile6], w[kRing6][kTile6], v[kRingV6][kTile6];
    unsigned char ys[2][kTile6];         // a chunk's outputs
    bf ops[2][4][kC6][PITCH];            // R~, K~, R0, K^ of this chunk and the next in turn
    uint64_t full[kRingV6];              // a chunk's raw rows have landed
    float wc[2][kN];                     // exp(c_C), or 0 when a start flag lies in the chunk
    float dpart[2][kC6][4];              // sum_i r u k per token over each warp's 16 channels
};
static_assert(4 * (sizeof(Fwd6cSmem) + 1024) <= 228 * 1024, "four CTAs per SM");

// Constant left operands (rows = token t, columns = token s; the two off-diagonal 8x8 blocks are zero) of the products with
// the log-decay rows that give, for every token and channel,
//   c_t - c_m (upto), c_{t-1} - c_m (before), and c_m | c_C - c_m (rows 0-7 | 8-15 of halves).
struct DecaySums {
    uint32_t upto_lo, upto_hi, before_lo, before_hi;
    __device__ __forceinline__ explicit DecaySums(int g, int q) {
        const int s = 2 * q;
        upto_lo = pack2(g < s ? -1.f : 0.f, g < s + 1 ? -1.f : 0.f);
        upto_hi = pack2(s <= g ? 1.f : 0.f, s + 1 <= g ? 1.f : 0.f);
        before_lo = pack2(g <= s ? -1.f : 0.f, g <= s + 1 ? -1.f : 0.f);
        before_hi = pack2(s < g ? 1.f : 0.f, s + 1 < g ? 1.f : 0.f);
    }
};
// Log-decay sums of a warp's 16 channels c0 .. c0 + 15: thread (g, q) gets, in x[nt][2 hh + e], the value of token g + 8 hh
// and channel c0 + 8 nt + 2 q + e.  wb: the raw rows as right operands (tokens 0-7 | 8-15 of channels 0-7, then 8-15).
__device__ __forceinline__ void decay_sums(const DecaySums& d, const uint32_t* wb, float (*upto)[4], float (*before)[4], float (*halves)[4]) {
    constexpr uint32_t kOnes = 0x3f803f80u;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
        for (int e = 0; e < 4; ++e) upto[nt][e] = before[nt][e] = halves[nt][e] = 0.f;
        mma_bf16(upto[nt], d.upto_lo, 0u, 0u, d.upto_hi, wb[2 * nt], wb[2 * nt + 1]);
        mma_bf16(before[nt], d.before_lo, 0u, 0u, d.before_hi, wb[2 * nt], wb[2 * nt + 1]);
        mma_bf16(halves[nt], kOnes, 0u, 0u, kOnes, wb[2 * nt], wb[2 * nt + 1]);
    }
}
// The same for a decay that is constant over the tokens: token x of the chunk counts if lo <= x < n.
__device__ __forceinline__ void decay_sums_const(const float* lw, int g, int lo, int n, float (*upto)[4], float (*before)[4], float (*halves)[4]) {
    auto count = [&](int t) { return min(max(t + 1 - lo, 0), max(n - lo, 0)); };     // tokens that count, up to t
    const int half = count(kC6 / 2 - 1), all = count(kC6 - 1);
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int t = g + 8 * (e >> 1);
            const float l = lw[2 * nt + (e & 1)];
            upto[nt][e] = l * (float)(count(t) - half);
            before[nt][e] = l * (float)(count(t - 1) - half);
            halves[nt][e] = l * (float)(e < 2 ? half : all - half);
        }
}
// both halves of a pair of bf16 at most zero (false for NaN)
__device__ __forceinline__ bool none_positive(uint32_t x) {
    return __hble2(*reinterpret_cast<const __nv_bfloat162*>(&x), __float2bfloat162_rn(0.f));
}
__device__ __forceinline__ float2 unpack2(uint32_t x) { return make_float2(__uint_as_float(x << 16), __uint_as_float(x & 0xffff0000u)); }
__device__ __forceinline__ void stmatrix_x4(void* row, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"((uint32_t)__cvta_generic_to_shared(row)),
                 "r"(r0), "r"(r1), "r"(r2), "r"(r3)
                 : "memory");
}
// an 8x8 tile, one pair of columns per lane, transposed inside the warp
__device__ __forceinline__ uint32_t transpose8x8(uint32_t a) {
    uint32_t d;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
    return d;
}

// start flags of a chunk as bits; no start in (s, t]
__device__ __forceinline__ bool same_segment(unsigned starts, int s, int t) { return ((starts & ((2u << t) - 1u)) >> (s + 1)) == 0; }

// One CTA of 128 threads per (batch, head).  ckpt: the state entering every chunk, bf16 S^T[value j][key i] in 8 column blocks
// of [64 j][8 i], and scores: every chunk's A^T as the left operand's words, lane by lane, for the backward (both NULL without one).  The kernel gives up (flag := ticket, see the file header) on a decay above 1
// and on a half-chunk decay beyond exp(-80).
__global__ void __launch_bounds__(128, 4)
wkv6_chunk_fwd_kernel(int Tlen, int H, const bf* __restrict__ r, const bf* __restrict__ k, const bf* __restrict__ v,
                      const bf* __restrict__ w, int w_per_token, const bf* __restrict__ u, const bf* __restrict__ s0,
                      const uint32_t* __restrict__ length, const uint8_t* __restrict__ new_starts, bf* __restrict__ y,
                      bf* __restrict__ s_out, bf* __restrict__ ckpt, uint4* __restrict__ scores, int* __restrict__ flag, int ticket,
                      int* __restrict__ residual_mark, const __grid_constant__ SeqMaps maps) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];   // (the swizzle is a function of the address)
    Fwd6cSmem& sm = *reinterpret_cast<Fwd6cSmem*>(smem_raw);
    const int bh = blockIdx.x, bi = bh / H, h = bh % H;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, q = lane & 3;
    const int j0 = warp * 16;                                    // this warp's value rows of S^T, and the channels it prepares
    const int frow = (lane & 15), fcol = (lane >> 4) * 8;        // a lane's row of a 16x16 block's four 8x8 tiles (ldmatrix, stmatrix)
    const size_t tok_stride = (size_t)H * kN;
    const size_t seq_base = (size_t)bi * Tlen * tok_stride + (size_t)h * kN;
    const size_t st_base = (size_t)bh * kN * kN;
    const int L = min((int)length[bi], Tlen);
    const int nC = (Tlen + kC6 - 1) / kC6;
    if (bh == 0 && tid == 0 && residual_mark != nullptr) *residual_mark = 0;   // chunked format (so far)
    const int c_out = L > 0 ? (L - 1) / kC6 : -1;                // the returned state leaves this chunk ...
    const int p_out = L > 0 ? (L - 1) % kC6 : -1;                // ... behind this token of it
    // A length inside a chunk: that chunk is walked in two parts, tokens 0..p_out and the rest, as if they were
    // two chunks (tokens outside the part at hand are inert: no decay, zero r and k, no output).
    const bool split = L > 0 && L < Tlen && p_out != kC6 - 1;

    // S^T tiles: acc[ni][e] = S[i = 8 ni + 2 q + (e & 1)][j = j0 + g + 8 (e >> 1)]
    float acc[8][4];
#pragma unroll
    for (int ni = 0; ni < 8; ++ni)
#pragma unroll
        for (int e = 0; e < 4; ++e)
            acc[ni][e] = __bfloat162float(s0[st_base + (size_t)(8 * ni + 2 * q + (e & 1)) * kN + j0 + g + 8 * (e >> 1)]);
    auto write_state = [&](bf* dst) {                             // [key i][value j], as the caller keeps it
#pragma unroll
        for (int ni = 0; ni < 8; ++ni)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                dst[st_base + (size_t)(8 * ni + 2 * q + (e & 1)) * kN + j0 + g + 8 * (e >> 1)] = __float2bfloat16_rn(acc[ni][e]);
    };
    if (L == 0) write_state(s_out);

    // raw rows by tiled copies, three chunks ahead (rows behind the sequence's end arrive as zeros)
    auto issue = [&](int c) {
        if (tid == 0 && c < nC) {
            uint64_t* bar = &sm.full[c % kRingV6];
            tc::mbar_expect_tx(bar, (w_per_token ? 4 : 3) * kTile6);
            tc::tensor_load_3d(sm.r[c % kRing6], &maps.m[0], h * kN, c * kC6, bi, bar);
            tc::tensor_load_3d(sm.k[c % kRing6], &maps.m[1], h * kN, c * kC6, bi, bar);
            tc::tensor_load_3d(sm.v[c % kRingV6], &maps.m[2], h * kN, c * kC6, bi, bar);
            if (w_per_token) tc::tensor_load_3d(sm.w[c % kRing6], &maps.m[3], h * kN, c * kC6, bi, bar);
        }
    };
    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < kRingV6; ++i) tc::mbar_init(&sm.full[i], 1);
        tc::mbar_init_fence();
    }
    __syncthreads();
    // this thread's places in a swizzled tile: its row of the warp's 16x16 block (matrix loads and stores), and the word of
    // channels j0 + 2 q, + 1 of token g (those of j0 + 8 + 2 q, + 1: XOR 16; token g + 8: + 1024)
    const int tile_row = frow * 128 + (((2 * warp + (lane >> 4)) ^ (frow & 7)) << 4);
    const int tile_word = g * 128 + (((2 * warp) ^ g) << 4) + 4 * q;
    // start flags: every warp fetches a chunk's sixteen for itself, two chunks ahead
    const uint8_t* const ns_row = new_starts + (size_t)bi * Tlen;
    auto load_ns = [&](int c) -> unsigned { return ns_row[min(c * kC6 + (lane & 15), Tlen - 1)]; };
    issue(0);
    issue(1);
    issue(2);
    unsigned ns_now = load_ns(0), ns_next = load_ns(1);

    float uu[4], lw_const[4];                                     // of channels j0 + 2 q, + 1, + 8, + 9
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const size_t at = (size_t)h * kN + j0 + 8 * (e >> 1) + 2 * q + (e & 1);
        uu[e] = __bfloat162float(u[at]);
        lw_const[e] = w_per_token ? 0.f : __logf(__bfloat162float(w[at]));
    }
    const DecaySums sums(g, q);
    bool good = true;

    // the chunk whose outputs wait in a tile: from token out_t on; a whole one leaves by a tiled copy, the parts of a split one
    // by rows out_lo .. out_hi - 1
    int out_t = -1, out_lo = 0, out_hi = kC6;
    auto send_outputs = [&](int buf) {
        if (out_t < 0) return;
        if (out_lo == 0 && out_hi == kC6) {
            if (tid == 0) {
                tc::tensor_store_3d(&maps.m[4], h * kN, out_t, bi, sm.ys[buf]);
                tc::bulk_commit();
            }
        } else {
            const int row = tid >> 3, piece = tid & 7;
            if (row >= out_lo && row < out_hi && out_t + row < Tlen)
                *reinterpret_cast<uint4*>(y + seq_base + (size_t)(out_t + row) * tok_stride + piece * 8) =
                    *reinterpret_cast<const uint4*>(sm.ys[buf] + row * 128 + ((piece ^ (row & 7)) << 4));
        }
    };
    // One chunk, or one part of the split chunk.  The two cases are separate instantiations: in the common one the
    // bounds of the part are the constants 0 and 16 and every test against them folds away.
    auto walk = [&](auto split_tag, const int c, const int buf, const int part_arg) {
        constexpr bool kSplitHere = decltype(split_tag)::value;
        const int part = kSplitHere ? part_arg : 0;
        const int lo = (kSplitHere && part == 1) ? p_out + 1 : 0, hi = (kSplitHere && part == 0) ? p_out + 1 : kC6;
        const int t0 = c * kC6, sl = c % kRing6;
        unsigned starts = __ballot_sync(0xffffffffu, ns_now != 0) & (0xffffu >> max(t0 + kC6 - Tlen, 0));
        if (kSplitHere) starts &= ((1u << hi) - 1u) & ~((1u << lo) - 1u);
        // ---- phase A: the scaled operands of this warp's channels
        if (!tc::mbar_wait(&sm.full[c % kRingV6], (c / kRingV6) & 1)) good = false;
        {
            float upto[2][4], before[2][4], halves[2][4];
            if (w_per_token) {
                uint32_t wb[4];
                ldmatrix_x4_trans(wb[0], wb[1], wb[2], wb[3], sm.w[sl] + tile_row);
                if (kSplitHere) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int s = 8 * (i & 1) + 2 * q;
                        wb[i] &= (s >= lo && s < hi ? 0xffffu : 0u) | (s + 1 >= lo && s + 1 < hi ? 0xffff0000u : 0u);
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) good = good && none_positive(wb[i]);   // a decay above 1 (or NaN) is outside what the scaling covers
                decay_sums(sums, wb, upto, before, halves);
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) good = good && lw_const[i] <= 0.f;
                decay_sums_const(lw_const, g, lo, min(hi, Tlen - t0), upto, before, halves);
            }
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) good = good && halves[nt][e] >= -kMaxHalfDecay;
            uint32_t rt[4], kt[4], r0[4], kh[4];                  // fragments, in the order (hh, nt) = 00, 10, 01, 11
            float dsum[2] = {0.f, 0.f};
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                const float2 em = make_float2(exp_fast(halves[nt][0]), exp_fast(halves[nt][1]));
                const float2 ecm = make_float2(exp_fast(halves[nt][2]), exp_fast(halves[nt][3]));
                if (g == 0)
                    *reinterpret_cast<float2*>(&sm.wc[buf][j0 + 8 * nt + 2 * q]) = starts == 0 ? make_float2(em.x * ecm.x, em.y * ecm.y) : make_float2(0.f, 0.f);
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int t = g + 8 * hh;
                    uint32_t rw = *reinterpret_cast<const uint32_t*>(sm.r[sl] + (tile_word ^ (16 * nt)) + 1024 * hh);
                    uint32_t kw = *reinterpret_cast<const uint32_t*>(sm.k[sl] + (tile_word ^ (16 * nt)) + 1024 * hh);
                    if (kSplitHere && !(t >= lo && t < hi)) rw = kw = 0;
                    const float2 rv = unpack2(rw), kv = unpack2(kw);
                    const float2 f2 = make_float2(exp_fast(before[nt][2 * hh]), exp_fast(before[nt][2 * hh + 1]));
                    const float2 f3 = make_float2(exp_fast(-upto[nt][2 * hh]), exp_fast(-upto[nt][2 * hh + 1]));
                    const int at = 2 * nt + hh;
                    rt[at] = pack2(rv.x * f2.x, rv.y * f2.y);
                    kt[at] = pack2(kv.x * f3.x, kv.y * f3.y);
                    r0[at] = pack2(rv.x * (f2.x * em.x), rv.y * (f2.y * em.y));
                    kh[at] = pack2(kv.x * (f3.x * ecm.x), kv.y * (f3.y * ecm.y));
                    dsum[hh] = fmaf(rv.x * uu[2 * nt], kv.x, fmaf(rv.y * uu[2 * nt + 1], kv.y, dsum[hh]));
                }
            }
            if (starts != 0) {     // tokens behind the first flag do not see S0, those in front of the last one do not reach S_C
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int t = g + 8 * hh;
                    const bool first = (starts & ((2u << t) - 1u)) == 0, last = (starts >> (t + 1)) == 0;
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) {
                        r0[2 * nt + hh] = first ? r0[2 * nt + hh] : 0u;
                        kh[2 * nt + hh] = last ? kh[2 * nt + hh] : 0u;
                    }
                }
            }
            stmatrix_x4(&sm.ops[buf][0][frow][j0 + fcol], rt[0], rt[1], rt[2], rt[3]);
            stmatrix_x4(&sm.ops[buf][1][frow][j0 + fcol], kt[0], kt[1], kt[2], kt[3]);
            stmatrix_x4(&sm.ops[buf][2][frow][j0 + fcol], r0[0], r0[1], r0[2], r0[3]);
            stmatrix_x4(&sm.ops[buf][3][frow][j0 + fcol], kh[0], kh[1], kh[2], kh[3]);
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                dsum[hh] += __shfl_xor_sync(0xffffffffu, dsum[hh], 1);
                dsum[hh] += __shfl_xor_sync(0xffffffffu, dsum[hh], 2);
                if (q == 0) sm.dpart[buf][g + 8 * hh][warp] = dsum[hh];
            }
        }
        if (tid == 0) tc::bulk_wait_read<0>();      // the outputs sent a chunk ago have left the tile that this chunk's go to
        tc::fence_async_smem();                     // (the previous chunk's outputs, for the copy that takes them)
        // the chunk's operands are complete; what the chunk before this one read behind its barrier (its v rows, the other
        // operand tiles) is free, and so are this chunk's r, k, w rows
        __syncthreads();
        if (!kSplitHere || part == 1) {
            issue(c + 3);
            ns_now = ns_next;
            ns_next = load_ns(c + 2);
        }
        send_outputs(buf ^ 1);
        out_t = t0;
        out_lo = lo;
        out_hi = hi;

        // ---- phase B: the products
        float yacc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};    // Y: rows token t, columns value j
        float sacc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};    // A: rows token t, columns token s
        bf* const dst = ckpt + ((size_t)bh * (nC + 1) + (part == 0 ? c : nC)) * kN * kN + (j0 + g) * 8 + 2 * q;
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
            Frag fr, f0, fk;
            ldmatrix_x4(fr.f[0], fr.f[1], fr.f[2], fr.f[3], &sm.ops[buf][0][frow][16 * ks + fcol]);
            ldmatrix_x4(fk.f[0], fk.f[1], fk.f[2], fk.f[3], &sm.ops[buf][1][frow][16 * ks + fcol]);
            ldmatrix_x4(f0.f[0], f0.f[1], f0.f[2], f0.f[3], &sm.ops[buf][2][frow][16 * ks + fcol]);
            // S^T tiles are right operands as they are: K = key channel (their columns), n = value row
            const uint32_t s00 = pack2(acc[2 * ks][0], acc[2 * ks][1]), s01 = pack2(acc[2 * ks + 1][0], acc[2 * ks + 1][1]);
            const uint32_t s10 = pack2(acc[2 * ks][2], acc[2 * ks][3]), s11 = pack2(acc[2 * ks + 1][2], acc[2 * ks + 1][3]);
            mma_bf16(yacc[0], f0.f[0], f0.f[1], f0.f[2], f0.f[3], s00, s01);
            mma_bf16(yacc[1], f0.f[0], f0.f[1], f0.f[2], f0.f[3], s10, s11);
            mma_ab(sacc[0], fr, fk, 0);
            mma_ab(sacc[1], fr, fk, 1);
            // the entering state for the backward (of the second part of a split chunk: slot nC), in 8 column blocks of
            // [64 rows j][8 keys i]: the eight row groups of a warp write one 128-byte line
            if (ckpt != nullptr) {
                *reinterpret_cast<uint32_t*>(dst + (2 * ks) * (kN * 8)) = s00;
                *reinterpret_cast<uint32_t*>(dst + (2 * ks) * (kN * 8) + 64) = s10;
                *reinterpret_cast<uint32_t*>(dst + (2 * ks + 1) * (kN * 8)) = s01;
                *reinterpret_cast<uint32_t*>(dst + (2 * ks + 1) * (kN * 8) + 64) = s11;
            }
        }
        uint32_t va[4];            // V^T of this warp: A fragments (M = value row, K = token), and V as right operands
        ldmatrix_x4_trans(va[0], va[2], va[1], va[3], sm.v[c % kRingV6] + tile_row);
        // strictly earlier tokens of the same segment; the diagonal is the u term.  (Rows and columns outside the part are zero
        // operands; the block of rows 0-7 and columns 8-15 is not used.)
        {
            const float4 d0 = *reinterpret_cast<const float4*>(&sm.dpart[buf][g][0]), d1 = *reinterpret_cast<const float4*>(&sm.dpart[buf][g + 8][0]);
            const float dg0 = (d0.x + d0.y) + (d0.z + d0.w), dg1 = (d1.x + d1.y) + (d1.z + d1.w);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int s = 2 * q + e;
                sacc[0][e] = s < g ? sacc[0][e] : (s == g ? dg0 : 0.f);
                sacc[1][2 + e] = s < g ? sacc[1][2 + e] : (s == g ? dg1 : 0.f);
            }
            if (starts != 0) {
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int s = 2 * q + e;
                    if (s < g && !same_segment(starts, s, g)) sacc[0][e] = 0.f;
                    if (!same_segment(starts, s, g + 8)) sacc[0][2 + e] = 0.f;
                    if (s < g && !same_segment(starts, s + 8, g + 8)) sacc[1][2 + e] = 0.f;
                }
            }
        }
        const uint32_t a0 = pack2(sacc[0][0], sacc[0][1]), a1 = pack2(sacc[0][2], sacc[0][3]), a3 = pack2(sacc[1][2], sacc[1][3]);
        if (scores != nullptr && warp == (c & 3))
            scores[((size_t)bh * (nC + 1) + (part == 0 ? c : nC)) * 32 + lane] = make_uint4(transpose8x8(a0), 0u, transpose8x8(a1), transpose8x8(a3));
        mma_bf16(yacc[0], a0, a1, 0u, a3, va[0], va[2]);
        mma_bf16(yacc[1], a0, a1, 0u, a3, va[1], va[3]);
        stmatrix_x4(sm.ys[buf] + tile_row, pack2(yacc[0][0], yacc[0][1]), pack2(yacc[0][2], yacc[0][3]), pack2(yacc[1][0], yacc[1][1]),
                    pack2(yacc[1][2], yacc[1][3]));
        // S^T <- S^T diag(exp(c_C)) [no start in the chunk] + V^T K^
#pragma unroll
        for (int np = 0; np < 4; ++np) {
            const float2 w0 = *reinterpret_cast<const float2*>(&sm.wc[buf][16 * np + 2 * q]);
            const float2 w1 = *reinterpret_cast<const float2*>(&sm.wc[buf][16 * np + 8 + 2 * q]);
            acc[2 * np][0] *= w0.x; acc[2 * np][1] *= w0.y; acc[2 * np][2] *= w0.x; acc[2 * np][3] *= w0.y;
            acc[2 * np + 1][0] *= w1.x; acc[2 * np + 1][1] *= w1.y; acc[2 * np + 1][2] *= w1.x; acc[2 * np + 1][3] *= w1.y;
            uint32_t b0, b1, b2, b3;        // key tiles 2 np (b0, b1) and 2 np + 1 (b2, b3)
            ldmatrix_x4_trans(b0, b1, b2, b3, &sm.ops[buf][3][frow][16 * np + fcol]);
            mma_bf16(acc[2 * np], va[0], va[1], va[2], va[3], b0, b1);
            mma_bf16(acc[2 * np + 1], va[0], va[1], va[2], va[3], b2, b3);
        }
        if (c == c_out && part == 0) write_state(s_out);
    };
    int buf = 0;
    for (int c = 0; c < nC; ++c) {
        if (split && c == c_out) {
#pragma unroll 1
            for (int part = 0; part < 2; ++part, buf ^= 1) walk(std::true_type{}, c, buf, part);
        } else {
            walk(std::false_type{}, c, buf, 0);
            buf ^= 1;
        }
    }
    tc::fence_async_smem();
    __syncthreads();
    send_outputs(buf ^ 1);
    if (tid == 0) tc::bulk_wait_read<0>();
    if (!good) atomicExch(flag, ticket);
}


// ------------------------------------------------------------------ backward --------
// Chunks in reverse order with the gradient of the state, dS^T[j][i], in accumulator tiles.  Per chunk, with the
// forward's operands rebuilt from the raw rows, and the entering state S0 and the scores A as the forward left them:
//     dA = mask(dY V^T)                                   dd_t = dy_t . v_t  (its diagonal, the u term)
//     dV  = A^T dY + K^ dS_C
//     dR~ = dY S0^T exp(c_m) + dA K~                      dK~ = V dS_C^T exp(c_C - c_m) + dA^T R~
//     dr = dR~ exp(c_{t-1} - c_m) + dd u k                dk = dK~ exp(c_m - c_s) + dd u r
//     dS0^T = dS_C^T diag(exp(c_C)) + dY^T R0
// and the gradient of the log-decay from the positions at which each factor depends on the cumulative sum:
//     dlw_tau = sum_{x >= tau} [ (r dr')_{x+1} - (k dk')_x ] + sum_s k dK^ exp(c_C - c_s) + exp(c_C) sum_j dS_C S0
// (dr', dk' without the u terms; dK^ = V dS_C^T; the two references to the middle cancel).
//
// Bound by instructions, as the forward, and split as it is: a warp prepares its 16 channels for all 16 tokens in fragment
// layout, and since that is also the layout of the gradients of those channels, the rows of r and k and the decay factors
// stay in its registers from the preparation to the results: nothing but operands and finished results passes through shared
// memory, the suffix sums over the tokens run over the lanes, and the sum over j of dS_C S0 is the diagonal of a product whose
// operands the other products load anyway (with dS_C as a high and a low bf16 part: the decay's gradient starts from this sum,
// and rounding dS_C once made it 4 % less accurate).  dA is computed by every warp for itself.  Two barriers per chunk.  At
// B=16, T=4096, H=32: 0.93 ms (1.56 ms with the factors, rows and sums exchanged through shared memory and four more score
// products per warp, which the forward now leaves).
struct BwdStage {
    unsigned char r[kTile6], k[kTile6], v[kTile6], w[kTile6], dy[kTile6];
    uint4 scores[32];          // A^T: the words of the left operand, lane by lane
    unsigned char pad[512];
    bf s0[8][kN][8];           // S0^T[j][i] as it lies in the residual: 8 column blocks of [64 rows j][8 keys i]
};
struct Bwd6cSmem {
    BwdStage st[2];
    unsigned char res[4][kTile6];   // dr, dk, dv, dw on their way out
    bf ops[4][kC6][PITCH];     // R~, K~ (each warp's own channels only), R0, K^
    bf ds[kN][PITCH];          // dS_C^T[j][i] in bf16, for the products that contract over j
    bf ds_low[kN][PITCH];      // and what that rounds off, for the sum that the decay's gradient starts from
    float wc[kN];              // exp(c_C), or 0 when a start flag lies in the chunk
    uint64_t full[2];
};
static_assert(sizeof(BwdStage) % 1024 == 0, "the swizzle is a function of the address");
static_assert(3 * (sizeof(Bwd6cSmem) + 1024) <= 228 * 1024, "three CTAs per SM");

__global__ void __launch_bounds__(128, 3)
wkv6_chunk_bwd_kernel(int Tlen, int H, const bf* __restrict__ u, const uint32_t* __restrict__ length, const uint8_t* __restrict__ new_starts, int has_dy, const bf* __restrict__ ds_out, const bf* __restrict__ ckpt, const uint4* __restrict__ scores,
                      const int* __restrict__ residual_mark, bf* __restrict__ dr, bf* __restrict__ dk, bf* __restrict__ dv,
                      bf* __restrict__ dw, float* __restrict__ du_head, bf* __restrict__ ds0,
                      int n_runs, int run_len, const bf* dsck, float* __restrict__ partial, int* __restrict__ status,
                      const __grid_constant__ SeqMaps maps) {
    let_next_in();
    if (word_behind(residual_mark) != 0) return;          // the forward fell back to the sequential kernels
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    Bwd6cSmem& sm = *reinterpret_cast<Bwd6cSmem*>(smem_raw);
    // n_runs > 1: a sequence is walked by n_runs CTAs, run rho = chunks [rho run_len, (rho + 1) run_len), each starting
    // from the state gradient that the carry kernel (wkv6_carry_bwd_kernel) left for the end of its run
    const int bh = blockIdx.x / n_runs, run = blockIdx.x % n_runs, bi = bh / H, h = bh % H;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, q = lane & 3;
    const int frow = (lane & 15), fcol = (lane >> 4) * 8;
    const int j0 = warp * 16;                 // value rows of dS^T, and channels of the token-by-channel results
    const size_t tok_stride = (size_t)H * kN;
    const size_t seq_base = (size_t)bi * Tlen * tok_stride + (size_t)h * kN;
    const size_t st_base = (size_t)bh * kN * kN;
    const int L = min((int)length[bi], Tlen);
    const int nC = (Tlen + kC6 - 1) / kC6;
    const int c_out = L > 0 ? (L - 1) / kC6 : -1, p_out = L > 0 ? (L - 1) % kC6 : -1;
    const bool split = L > 0 && L < Tlen && p_out != kC6 - 1;      // see the forward: that chunk is walked in two parts
    const int c_lo = run * run_len, c_hi = min(nC, c_lo + run_len);
    if (c_lo >= c_hi) return;

    auto issue = [&](int c, int stage) {
        if (tid == 0 && c >= c_lo) {
            BwdStage& st = sm.st[stage];
            uint64_t* bar = &sm.full[stage];
            tc::mbar_expect_tx(bar, (4 + has_dy) * kTile6 + sizeof(st.s0) + sizeof(st.scores));
            tc::tensor_load_3d(st.r, &maps.m[0], h * kN, c * kC6, bi, bar);
            tc::tensor_load_3d(st.k, &maps.m[1], h * kN, c * kC6, bi, bar);
            tc::tensor_load_3d(st.v, &maps.m[2], h * kN, c * kC6, bi, bar);
            tc::tensor_load_3d(st.w, &maps.m[3], h * kN, c * kC6, bi, bar);
            if (has_dy) tc::tensor_load_3d(st.dy, &maps.m[4], h * kN, c * kC6, bi, bar);
            tc::bulk_load(st.s0, ckpt + ((size_t)bh * (nC + 1) + c) * kN * kN, sizeof(st.s0), bar);
            tc::bulk_load(st.scores, scores + ((size_t)bh * (nC + 1) + c) * 32, sizeof(st.scores), bar);
        }
    };
    if (tid == 0) {
        tc::mbar_init(&sm.full[0], 1);
        tc::mbar_init(&sm.full[1], 1);
        tc::mbar_init_fence();
    }
    if (!has_dy)
#pragma unroll
        for (int stg = 0; stg < 2; ++stg) *reinterpret_cast<uint4*>(sm.st[stg].dy + tid * 16) = make_uint4(0, 0, 0, 0);
    __syncthreads();
    issue(c_hi - 1, 0);
    const uint8_t* const ns_row = new_starts + (size_t)bi * Tlen;
    auto load_ns = [&](int c) -> unsigned { return ns_row[min(max(c, 0) * kC6 + (lane & 15), Tlen - 1)]; };
    unsigned ns_now = load_ns(c_hi - 1), ns_next = load_ns(c_hi - 2);

    float acc[8][4];
    if (run == n_runs - 1 || c_hi >= nC) {
#pragma unroll
        for (int ni = 0; ni < 8; ++ni)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[ni][e] = 0.f;
    } else {
        const bf* src = dsck + ((size_t)bh * n_runs + run) * kN * kN;
#pragma unroll
        for (int ni = 0; ni < 8; ++ni) {
            const float2 lo2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(src + (size_t)(j0 + g) * kN + 8 * ni + 2 * q));
            const float2 hi2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(src + (size_t)(j0 + g + 8) * kN + 8 * ni + 2 * q));
            acc[ni][0] = lo2.x; acc[ni][1] = lo2.y; acc[ni][2] = hi2.x; acc[ni][3] = hi2.y;
        }
    }
    auto add_ds_out = [&]() {
        if (ds_out == nullptr) return;
#pragma unroll
        for (int ni = 0; ni < 8; ++ni)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                acc[ni][e] += __bfloat162float(ds_out[st_base + (size_t)(8 * ni + 2 * q + (e & 1)) * kN + j0 + g + 8 * (e >> 1)]);
    };
    // the state entering a part of the split chunk and the part's scores, fetched on the spot (once or twice per sequence)
    auto fetch_state = [&](int slot, int stage) {
        const uint4* src = reinterpret_cast<const uint4*>(ckpt + ((size_t)bh * (nC + 1) + slot) * kN * kN);
        uint4* dst = reinterpret_cast<uint4*>(&sm.st[stage].s0[0][0][0]);
        __syncthreads();
#pragma unroll
        for (int rr = 0; rr < 4; ++rr) dst[tid + 128 * rr] = src[tid + 128 * rr];
        if (warp == 0) sm.st[stage].scores[lane] = scores[((size_t)bh * (nC + 1) + slot) * 32 + lane];
        __syncthreads();
    };

    float uu[4];                                                  // of channels j0 + 2 q, + 1, + 8, + 9
#pragma unroll
    for (int e = 0; e < 4; ++e) uu[e] = __bfloat162float(u[(size_t)h * kN + j0 + 8 * (e >> 1) + 2 * q + (e & 1)]);
    const DecaySums sums(g, q);
    const int tile_row = frow * 128 + (((2 * warp + (lane >> 4)) ^ (frow & 7)) << 4);      // as in the forward
    const int tile_word = g * 128 + (((2 * warp) ^ g) << 4) + 4 * q;
    float du_acc[4] = {0.f, 0.f, 0.f, 0.f};    // this thread's tokens of those channels
    bool waited = true;

    // the chunk whose results wait in the result tiles (see send_outputs of the forward)
    int out_t = -1, out_lo = 0, out_hi = kC6;
    auto send_results = [&]() {
        if (out_t < 0) return;
        if (out_lo == 0 && out_hi == kC6) {
            if (tid == 0) {
                tc::tensor_store_3d(&maps.m[5], h * kN, out_t, bi, sm.res[0]);
                tc::tensor_store_3d(&maps.m[6], h * kN, out_t, bi, sm.res[1]);
                tc::tensor_store_3d(&maps.m[7], h * kN, out_t, bi, sm.res[2]);
                tc::tensor_store_3d(&maps.m[8], h * kN, out_t, bi, sm.res[3]);
                tc::bulk_commit();
            }
        } else {
            const int row = tid >> 3, piece = tid & 7;
            if (row >= out_lo && row < out_hi && out_t + row < Tlen) {
                const size_t off = seq_base + (size_t)(out_t + row) * tok_stride + piece * 8;
                const int at = row * 128 + ((piece ^ (row & 7)) << 4);
                *reinterpret_cast<uint4*>(dr + off) = *reinterpret_cast<const uint4*>(sm.res[0] + at);
                *reinterpret_cast<uint4*>(dk + off) = *reinterpret_cast<const uint4*>(sm.res[1] + at);
                *reinterpret_cast<uint4*>(dv + off) = *reinterpret_cast<const uint4*>(sm.res[2] + at);
                *reinterpret_cast<uint4*>(dw + off) = *reinterpret_cast<const uint4*>(sm.res[3] + at);
            }
        }
    };
    auto walk = [&](auto split_tag, const int c, const int it, const int part_arg) {
        constexpr bool kSplitHere = decltype(split_tag)::value;
        const int part = kSplitHere ? part_arg : 0;
        const int stage = it & 1;
        BwdStage& st = sm.st[stage];
        const int lo = (kSplitHere && part == 1) ? p_out + 1 : 0, hi = (kSplitHere && part == 0) ? p_out + 1 : kC6;
        const int t0 = c * kC6;
        const bool first_visit = !kSplitHere || part == 1;
        if (first_visit) issue(c - 1, stage ^ 1);
        unsigned starts = __ballot_sync(0xffffffffu, ns_now != 0) & (0xffffu >> max(t0 + kC6 - Tlen, 0));
        if (kSplitHere) starts &= ((1u << hi) - 1u) & ~((1u << lo) - 1u);
        if (!kSplitHere || part == 0) {
            ns_now = ns_next;
            ns_next = load_ns(c - 2);
        }
        if (!tc::mbar_wait(&sm.full[stage], (it >> 1) & 1)) waited = false;
        if (kSplitHere) fetch_state(part == 1 ? nC : c, stage);       // (slot nC: the state behind token p_out)
        if (c == c_out && part == 0) add_ds_out();

        // ---- phase A: dS_C^T in bf16; the scaled operands of this warp's channels, as in the forward
        uint32_t dsp[8][2];                   // [ni][value rows g | g + 8]
#pragma unroll
        for (int ni = 0; ni < 8; ++ni) {
            dsp[ni][0] = pack2(acc[ni][0], acc[ni][1]);
            dsp[ni][1] = pack2(acc[ni][2], acc[ni][3]);
        }
#pragma unroll
        for (int np = 0; np < 4; ++np) stmatrix_x4(&sm.ds[j0 + frow][16 * np + fcol], dsp[2 * np][0], dsp[2 * np][1], dsp[2 * np + 1][0], dsp[2 * np + 1][1]);
#pragma unroll
        for (int np = 0; np < 4; ++np) {
            uint32_t low[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int ni = 2 * np + (i >> 1), half = i & 1;
                const float2 high = unpack2(dsp[ni][half]);
                low[i] = pack2(acc[ni][2 * half] - high.x, acc[ni][2 * half + 1] - high.y);
            }
            stmatrix_x4(&sm.ds_low[j0 + frow][16 * np + fcol], low[0], low[1], low[2], low[3]);
        }
        uint32_t rw[4], kw[4];                // raw rows, [2 nt + hh]
        float2 f2[4], f3[4], em[2], ecm[2];   // what turns dR~, dK~ into dr, dk; and dR0, dK^ into dR~, dK~
        {
            float upto[2][4], before[2][4], halves[2][4];
            uint32_t wb[4];
            ldmatrix_x4_trans(wb[0], wb[1], wb[2], wb[3], st.w + tile_row);
            if (kSplitHere) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int s = 8 * (i & 1) + 2 * q;
                    wb[i] &= (s >= lo && s < hi ? 0xffffu : 0u) | (s + 1 >= lo && s + 1 < hi ? 0xffff0000u : 0u);
                }
            }
            decay_sums(sums, wb, upto, before, halves);
            uint32_t rt[4], kt[4], r0[4], kh[4];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                em[nt] = make_float2(exp_fast(halves[nt][0]), exp_fast(halves[nt][1]));
                ecm[nt] = make_float2(exp_fast(halves[nt][2]), exp_fast(halves[nt][3]));
                if (g == 0)
                    *reinterpret_cast<float2*>(&sm.wc[j0 + 8 * nt + 2 * q]) = starts == 0 ? make_float2(em[nt].x * ecm[nt].x, em[nt].y * ecm[nt].y) : make_float2(0.f, 0.f);
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int at = 2 * nt + hh, t = g + 8 * hh;
                    rw[at] = *reinterpret_cast<const uint32_t*>(st.r + (tile_word ^ (16 * nt)) + 1024 * hh);
                    kw[at] = *reinterpret_cast<const uint32_t*>(st.k + (tile_word ^ (16 * nt)) + 1024 * hh);
                    if (kSplitHere && !(t >= lo && t < hi)) rw[at] = kw[at] = 0;
                    const float2 rv = unpack2(rw[at]), kv = unpack2(kw[at]);
                    f2[at] = make_float2(exp_fast(before[nt][2 * hh]), exp_fast(before[nt][2 * hh + 1]));
                    f3[at] = make_float2(exp_fast(-upto[nt][2 * hh]), exp_fast(-upto[nt][2 * hh + 1]));
                    rt[at] = pack2(rv.x * f2[at].x, rv.y * f2[at].y);
                    kt[at] = pack2(kv.x * f3[at].x, kv.y * f3[at].y);
                    r0[at] = pack2(rv.x * (f2[at].x * em[nt].x), rv.y * (f2[at].y * em[nt].y));
                    kh[at] = pack2(kv.x * (f3[at].x * ecm[nt].x), kv.y * (f3[at].y * ecm[nt].y));
                }
            }
            if (starts != 0) {
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int t = g + 8 * hh;
                    const bool first = (starts & ((2u << t) - 1u)) == 0, last = (starts >> (t + 1)) == 0;
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) {
                        r0[2 * nt + hh] = first ? r0[2 * nt + hh] : 0u;
                        kh[2 * nt + hh] = last ? kh[2 * nt + hh] : 0u;
                    }
                }
            }
            stmatrix_x4(&sm.ops[0][frow][j0 + fcol], rt[0], rt[1], rt[2], rt[3]);
            stmatrix_x4(&sm.ops[1][frow][j0 + fcol], kt[0], kt[1], kt[2], kt[3]);
            stmatrix_x4(&sm.ops[2][frow][j0 + fcol], r0[0], r0[1], r0[2], r0[3]);
            stmatrix_x4(&sm.ops[3][frow][j0 + fcol], kh[0], kh[1], kh[2], kh[3]);
        }
        tc::fence_async_smem();               // (the previous chunk's results, for the copies that take them)
        __syncthreads();                      // the operands are complete
        send_results();

        // ---- phase B: the products
        float dA[2][4];                       // t x s
        float dR[2][4], dK[2][4], dV[2][4];   // token x this warp's 16 channels (dV: its value columns)
        float dot[2][4];                      // its diagonals: sum_j dS_C S0 of channels j0 + g (tile 0) and j0 + 8 + g (tile 1)
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) dA[nt][e] = dR[nt][e] = dK[nt][e] = dV[nt][e] = dot[nt][e] = 0.f;
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
            Frag fdy, fv, fh, fs, fd, fl;
            const int row_at = frow * 128 + (((2 * ks + (lane >> 4)) ^ (frow & 7)) << 4);
            ldmatrix_x4(fdy.f[0], fdy.f[1], fdy.f[2], fdy.f[3], st.dy + row_at);
            ldmatrix_x4(fv.f[0], fv.f[1], fv.f[2], fv.f[3], st.v + row_at);
            ldmatrix_x4(fh.f[0], fh.f[1], fh.f[2], fh.f[3], &sm.ops[3][frow][16 * ks + fcol]);
            // [value j][channel i] tiles as right operands (K = j); as left operands their transposes are the same words
            ldmatrix_x4_trans(fs.f[0], fs.f[1], fs.f[2], fs.f[3], &st.s0[j0 / 8 + (lane >> 4)][16 * ks + frow][0]);
            ldmatrix_x4_trans(fd.f[0], fd.f[1], fd.f[2], fd.f[3], &sm.ds[16 * ks + frow][j0 + fcol]);
            ldmatrix_x4_trans(fl.f[0], fl.f[1], fl.f[2], fl.f[3], &sm.ds_low[16 * ks + frow][j0 + fcol]);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                mma_ab(dA[nt], fdy, fv, nt);
                mma_bf16(dR[nt], fdy.f[0], fdy.f[1], fdy.f[2], fdy.f[3], fs.f[2 * nt], fs.f[2 * nt + 1]);
                mma_bf16(dK[nt], fv.f[0], fv.f[1], fv.f[2], fv.f[3], fd.f[2 * nt], fd.f[2 * nt + 1]);
                // dS_C^T tiles as right operand: K = key channel (their columns), n = value row (their rows)
                mma_bf16(dV[nt], fh.f[0], fh.f[1], fh.f[2], fh.f[3], dsp[2 * ks][nt], dsp[2 * ks + 1][nt]);
                mma_bf16(dot[nt], fs.f[0], fs.f[2], fs.f[1], fs.f[3], fd.f[2 * nt], fd.f[2 * nt + 1]);
                mma_bf16(dot[nt], fs.f[0], fs.f[2], fs.f[1], fs.f[3], fl.f[2 * nt], fl.f[2 * nt + 1]);
            }
        }
        // dd of this thread's two token rows: the diagonal of dA sits in lane 4 g + g / 2
        float dd[2];
        {
            const int src = (lane & ~3) | (g >> 1);
            dd[0] = __shfl_sync(0xffffffffu, (g & 1) ? dA[0][1] : dA[0][0], src);
            dd[1] = __shfl_sync(0xffffffffu, (g & 1) ? dA[1][3] : dA[1][2], src);
        }
        // masks: pairs s < t of one segment (the block t < 8 <= s is not used)
        {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int col = 2 * q + e;
                dA[0][e] = col < g ? dA[0][e] : 0.f;
                dA[1][2 + e] = col < g ? dA[1][2 + e] : 0.f;
            }
            if (starts != 0) {
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int col = 2 * q + e;
                    if (col < g && !same_segment(starts, col, g)) dA[0][e] = 0.f;
                    if (!same_segment(starts, col, g + 8)) dA[0][2 + e] = 0.f;
                    if (col < g && !same_segment(starts, col + 8, g + 8)) dA[1][2 + e] = 0.f;
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {          // S0 reaches the tokens in front of the first flag, S_C holds those from the last one on
                    const int t = g + 8 * (e >> 1);
                    const bool first = (starts & ((2u << t) - 1u)) == 0, last = (starts >> (t + 1)) == 0;
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) {
                        dR[nt][e] = first ? dR[nt][e] : 0.f;
                        dK[nt][e] = last ? dK[nt][e] : 0.f;
                    }
                }
            }
        }
        uint32_t yf[4];                       // dY of this warp's value columns, transposed: (tokens 0-7 | 8-15) of columns 0-7, then 8-15
        ldmatrix_x4_trans(yf[0], yf[1], yf[2], yf[3], st.dy + tile_row);
        {   // dV += A^T dY
            const uint4 at = st.scores[lane];
            mma_bf16(dV[0], at.x, 0u, at.z, at.w, yf[0], yf[1]);
            mma_bf16(dV[1], at.x, 0u, at.z, at.w, yf[2], yf[3]);
        }
        float lump[4];                        // per channel: sum_s k dK^ exp(c_C - c_s) over this thread's tokens
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float m = e ? em[nt].y : em[nt].x, mc = e ? ecm[nt].y : ecm[nt].x;
                float sum = 0.f;
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int at = 2 * nt + hh;
                    dR[nt][2 * hh + e] *= m;
                    dK[nt][2 * hh + e] *= mc;
                    const float kv = e ? unpack2(kw[at]).y : unpack2(kw[at]).x;
                    sum = fmaf(kv * (e ? f3[at].y : f3[at].x), dK[nt][2 * hh + e], sum);
                }
                lump[2 * nt + e] = sum;
            }
        }
        {   // dR~ += dA K~, dK~ += dA^T R~
            const uint32_t a0 = pack2(dA[0][0], dA[0][1]), a1 = pack2(dA[0][2], dA[0][3]), a3 = pack2(dA[1][2], dA[1][3]);
            uint32_t b0, b1, b2, b3;
            ldmatrix_x4_trans(b0, b1, b2, b3, &sm.ops[1][frow][j0 + fcol]);
            mma_bf16(dR[0], a0, a1, 0u, a3, b0, b1);
            mma_bf16(dR[1], a0, a1, 0u, a3, b2, b3);
            ldmatrix_x4_trans(b0, b1, b2, b3, &sm.ops[0][frow][j0 + fcol]);
            const uint32_t t0_ = transpose8x8(a0), t2 = transpose8x8(a1), t3 = transpose8x8(a3);
            mma_bf16(dK[0], t0_, 0u, t2, t3, b0, b1);
            mma_bf16(dK[1], t0_, 0u, t2, t3, b2, b3);
        }
        // + exp(c_C) sum_j dS_C S0, from the lanes that hold the diagonals (as one of the sum's eight summands, below)
        {
            const float d0 = __shfl_sync(0xffffffffu, dot[0][0], 9 * q), d1 = __shfl_sync(0xffffffffu, dot[0][1], 9 * q + 4);
            const float d2 = __shfl_sync(0xffffffffu, dot[1][2], 9 * q), d3 = __shfl_sync(0xffffffffu, dot[1][3], 9 * q + 4);
            if (g == 0) {
                const float2 w0 = *reinterpret_cast<const float2*>(&sm.wc[j0 + 2 * q]), w1 = *reinterpret_cast<const float2*>(&sm.wc[j0 + 8 + 2 * q]);
                lump[0] = fmaf(d0, w0.x, lump[0]);
                lump[1] = fmaf(d1, w0.y, lump[1]);
                lump[2] = fmaf(d2, w1.x, lump[2]);
                lump[3] = fmaf(d3, w1.y, lump[3]);
            }
        }
        // ---- dS0^T = dS_C^T diag(exp(c_C)) [no start in the chunk] + dY^T R0
#pragma unroll
        for (int np = 0; np < 4; ++np) {
            const float2 w0 = *reinterpret_cast<const float2*>(&sm.wc[16 * np + 2 * q]);
            const float2 w1 = *reinterpret_cast<const float2*>(&sm.wc[16 * np + 8 + 2 * q]);
            acc[2 * np][0] *= w0.x; acc[2 * np][1] *= w0.y; acc[2 * np][2] *= w0.x; acc[2 * np][3] *= w0.y;
            acc[2 * np + 1][0] *= w1.x; acc[2 * np + 1][1] *= w1.y; acc[2 * np + 1][2] *= w1.x; acc[2 * np + 1][3] *= w1.y;
            uint32_t b0, b1, b2, b3;
            ldmatrix_x4_trans(b0, b1, b2, b3, &sm.ops[2][frow][16 * np + fcol]);
            mma_bf16(acc[2 * np], yf[0], yf[2], yf[1], yf[3], b0, b1);
            mma_bf16(acc[2 * np + 1], yf[0], yf[2], yf[1], yf[3], b2, b3);
        }
        if (tid == 0) tc::bulk_wait_read<0>();      // the previous chunk's results have left the result tiles
        __syncthreads();                            // nobody reads this chunk's tiles any more
        // ---- epilogue
        uint32_t rdr[4], rdk[4], rdw[4];
        float dlw[2][4];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            float ea[2][2], z[2][2];                // [hh][column]: r dr', and r dr' - k dk'
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const int at = 2 * nt + hh, e0 = 2 * hh;
                const float2 rv = unpack2(rw[at]), kv = unpack2(kw[at]);
                const float drx = dR[nt][e0] * f2[at].x, dry = dR[nt][e0 + 1] * f2[at].y;
                const float dkx = dK[nt][e0] * f3[at].x, dky = dK[nt][e0 + 1] * f3[at].y;
                const float dux = dd[hh] * uu[2 * nt], duy = dd[hh] * uu[2 * nt + 1];
                rdr[at] = pack2(fmaf(dux, kv.x, drx), fmaf(duy, kv.y, dry));
                rdk[at] = pack2(fmaf(dux, rv.x, dkx), fmaf(duy, rv.y, dky));
                ea[hh][0] = rv.x * drx;
                ea[hh][1] = rv.y * dry;
                z[hh][0] = ea[hh][0] - kv.x * dkx;
                z[hh][1] = ea[hh][1] - kv.y * dky;
                du_acc[2 * nt] = fmaf(dd[hh] * rv.x, kv.x, du_acc[2 * nt]);
                du_acc[2 * nt + 1] = fmaf(dd[hh] * rv.y, kv.y, du_acc[2 * nt + 1]);
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                // sums over the tokens from each on (lanes g, g + 1, ..., 7 of both halves), and of `lump` over all lanes
                float s0_ = z[0][e], s1 = z[1][e], l = lump[2 * nt + e];
#pragma unroll
                for (int d = 1; d < 8; d <<= 1) {
                    const float a = __shfl_down_sync(0xffffffffu, s0_, 4 * d), b = __shfl_down_sync(0xffffffffu, s1, 4 * d);
                    s0_ += g + d < 8 ? a : 0.f;
                    s1 += g + d < 8 ? b : 0.f;
                    l += __shfl_xor_sync(0xffffffffu, l, 4 * d);
                }
                s0_ += __shfl_sync(0xffffffffu, s1, q);        // the second half's total
                dlw[nt][e] = s0_ - ea[0][e] + l;
                dlw[nt][2 + e] = s1 - ea[1][e] + l;
            }
        }
        stmatrix_x4(sm.res[0] + tile_row, rdr[0], rdr[1], rdr[2], rdr[3]);
        stmatrix_x4(sm.res[1] + tile_row, rdk[0], rdk[1], rdk[2], rdk[3]);
        stmatrix_x4(sm.res[2] + tile_row, pack2(dV[0][0], dV[0][1]), pack2(dV[0][2], dV[0][3]), pack2(dV[1][0], dV[1][1]), pack2(dV[1][2], dV[1][3]));
#pragma unroll
        for (int at = 0; at < 4; ++at) rdw[at] = pack2(dlw[at >> 1][2 * (at & 1)], dlw[at >> 1][2 * (at & 1) + 1]);
        stmatrix_x4(sm.res[3] + tile_row, rdw[0], rdw[1], rdw[2], rdw[3]);
        out_t = t0;
        out_lo = lo;
        out_hi = hi;
    };
    for (int c = c_hi - 1, it = 0; c >= c_lo; --c, ++it) {
        if (split && c == c_out) {
#pragma unroll 1
            for (int part = 1; part >= 0; --part) walk(std::true_type{}, c, it, part);   // tokens behind `length` first
        } else {
            walk(std::false_type{}, c, it, 0);
        }
    }
    tc::fence_async_smem();
    __syncthreads();
    send_results();
    if (tid == 0) tc::bulk_wait_read<0>();
    if (run == 0) {
        if (L == 0) add_ds_out();
#pragma unroll
        for (int ni = 0; ni < 8; ++ni)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                ds0[st_base + (size_t)(8 * ni + 2 * q + (e & 1)) * kN + j0 + g + 8 * (e >> 1)] = __float2bfloat16_rn(acc[ni][e]);
    }
    // du of the (batch, head), or this run's share for the reduction behind the kernel: the sum over this thread's token rows,
    // then over the eight row groups of the warp
    float* const du_dst = n_runs == 1 ? du_head + (size_t)bh * kN : partial + ((size_t)bh * n_runs + run) * kN;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        float p = du_acc[e];
#pragma unroll
        for (int m = 4; m < 32; m <<= 1) p += __shfl_xor_sync(0xffffffffu, p, m);
        if (g == 0) du_dst[j0 + 8 * (e >> 1) + 2 * q + (e & 1)] = p;
    }
    if (!waited && status != nullptr) atomicExch(status, 5);
}

// ------------------------------------------------------------------ the state-gradient carry
// The only part of the backward that is sequential in T, on its own: dS0^T = dS_C^T diag(exp(c_C)) [no start in the
// chunk] + dY^T R0 per chunk (and the cotangent of the returned state where it enters), with dS^T in accumulator
// registers.  It leaves the state gradient at the end of every run of `run_len` chunks, from which the gradient kernel
// above walks the runs in parallel.
// Unlike the other kernels of this file it walks 64 tokens at a time: it uses no factor other than exp(cumulative
// log-decay) <= 1, so nothing limits its chunk, and a quarter of the steps means a quarter of the barriers and waits.  The
// operands are prepared as in the forward, a warp its 16 channels, R0 in place over the r rows: two 24 KB stages, four CTAs
// per SM, which 512 sequences need to run at once.  B=16, T=4096, H=32: 0.153 ms (0.257 ms with sums as a scan over
// quarters of the step and rows fetched by every thread), 0.8 GB at 5.3 TB/s.
constexpr int kCB = 64;            // tokens per step of the carry
constexpr int kCarryStages = 2;
constexpr int kTileCB = kCB * kN * 2;
static_assert(kRunLen6 % (kCB / kC6) == 0, "runs must end at a step of the carry");
struct Carry6Smem {
    unsigned char r[kCarryStages][kTileCB], w[kCarryStages][kTileCB], dy[kCarryStages][kTileCB];
    float wc[kN];                  // exp(c_C), or 0 when a start flag lies in the step
    uint64_t full[kCarryStages];
};
static_assert(4 * (sizeof(Carry6Smem) + 1024) <= 228 * 1024, "four CTAs per SM");

__global__ void __launch_bounds__(128, 4)
wkv6_carry_bwd_kernel(int Tlen, int H, const bf* __restrict__ r, const uint32_t* __restrict__ length,
                      const uint8_t* __restrict__ new_starts, int has_dy, const bf* __restrict__ ds_out,
                      const int* __restrict__ residual_mark, int n_runs, int run_len, bf* __restrict__ dsck, int* __restrict__ status,
                      const __grid_constant__ SeqMaps maps) {
    let_next_in();
    if (*residual_mark != 0) return;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    Carry6Smem& sm = *reinterpret_cast<Carry6Smem*>(smem_raw);
    const int bh = blockIdx.x, bi = bh / H, h = bh % H;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, q = lane & 3;
    const int frow = lane & 15;
    const int j0 = warp * 16;
    const size_t tok_stride = (size_t)H * kN;
    const size_t seq_base = (size_t)bi * Tlen * tok_stride + (size_t)h * kN;
    const size_t st_base = (size_t)bh * kN * kN;
    const int L = min((int)length[bi], Tlen);
    const int nB = (Tlen + kCB - 1) / kCB;                 // steps of the carry
    const int run_steps = run_len / (kCB / kC6);           // steps per run of the gradient kernel
    const int c_out = L > 0 ? (L - 1) / kCB : -1, p_out = L > 0 ? (L - 1) % kCB : -1;
    const bool split = L > 0 && L < Tlen && p_out != kCB - 1;
    const int c_stop = run_steps;      // nothing below the first run's end is needed: run 0 starts from the state left there

    float acc[8][4];
#pragma unroll
    for (int ni = 0; ni < 8; ++ni)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[ni][e] = 0.f;
    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < kCarryStages; ++i) tc::mbar_init(&sm.full[i], 1);
        tc::mbar_init_fence();
    }
    __syncthreads();
    auto issue = [&](int c) {          // step c, the (nB - 1 - c)th
        if (tid == 0 && c >= c_stop) {
            const int stage = (nB - 1 - c) % kCarryStages;
            uint64_t* bar = &sm.full[stage];
            tc::mbar_expect_tx(bar, (2 + has_dy) * kTileCB);
            tc::tensor_load_3d(sm.r[stage], &maps.m[0], h * kN, c * kCB, bi, bar);
            tc::tensor_load_3d(sm.w[stage], &maps.m[1], h * kN, c * kCB, bi, bar);
            if (has_dy) tc::tensor_load_3d(sm.dy[stage], &maps.m[2], h * kN, c * kCB, bi, bar);
        }
    };
    issue(nB - 1);
    const uint8_t* const ns_row = new_starts + (size_t)bi * Tlen;
    auto load_ns = [&](int c, int half) -> unsigned { return ns_row[min(max(c, 0) * kCB + 32 * half + lane, Tlen - 1)]; };
    unsigned ns_lo = load_ns(nB - 1, 0), ns_hi = load_ns(nB - 1, 1);
    // places in a swizzled tile, as in the forward; of a 16x16 block's rows in column piece 2 x, + 1
    auto block_row = [&](int x) { return frow * 128 + (((2 * x + (lane >> 4)) ^ (frow & 7)) << 4); };
    const int tile_row = block_row(warp);
    const int tile_word = g * 128 + (((2 * warp) ^ g) << 4) + 4 * q;
    // constant left operands: strictly earlier tokens of a 16-token block, and all of them
    const uint32_t earlier = pack2(2 * q < g ? 1.f : 0.f, 2 * q + 1 < g ? 1.f : 0.f);
    constexpr uint32_t kOnes = 0x3f803f80u;
    bool waited = true;

    auto walk = [&](auto split_tag, const int c, const int part_arg) {
        constexpr bool kSplitHere = decltype(split_tag)::value;
        const int part = kSplitHere ? part_arg : 0;
        const int lo = (kSplitHere && part == 1) ? p_out + 1 : 0, hi = (kSplitHere && part == 0) ? p_out + 1 : kCB;
        const int it = nB - 1 - c, stage = it % kCarryStages;
        const int t0 = c * kCB;
        unsigned long long starts = (unsigned long long)__ballot_sync(0xffffffffu, ns_lo != 0) | (unsigned long long)__ballot_sync(0xffffffffu, ns_hi != 0) << 32;
        starts &= ~0ull >> max(t0 + kCB - Tlen, 0);
        if (kSplitHere) starts &= (hi < kCB ? (1ull << hi) - 1ull : ~0ull) & ~((1ull << lo) - 1ull);
        tc::fence_async_smem();       // (R0 was written over the r rows that the next copy replaces)
        __syncthreads();              // the tiles of step c + 1 are no longer read
        if (!kSplitHere || part == 1) {
            issue(c - 1);
            if (!tc::mbar_wait(&sm.full[stage], (it / kCarryStages) & 1)) waited = false;
        } else {
            // the first visit turned r into R0 in place: fetch the rows again for the part in front of `length`
#pragma unroll
            for (int rr = 0; rr < kCB / 16; ++rr) {
                const int row = (tid >> 3) + 16 * rr, piece = tid & 7;
                *reinterpret_cast<uint4*>(sm.r[stage] + row * 128 + ((piece ^ (row & 7)) << 4)) =
                    t0 + row < Tlen ? *reinterpret_cast<const uint4*>(r + seq_base + (size_t)(t0 + row) * tok_stride + piece * 8) : make_uint4(0, 0, 0, 0);
            }
            __syncthreads();
        }
        if (!kSplitHere || part == 0) {
            ns_lo = load_ns(c - 1, 0);
            ns_hi = load_ns(c - 1, 1);
        }
        if (c == c_out && part == 0 && ds_out != nullptr) {
#pragma unroll
            for (int ni = 0; ni < 8; ++ni)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    acc[ni][e] += __bfloat162float(ds_out[st_base + (size_t)(8 * ni + 2 * q + (e & 1)) * kN + j0 + g + 8 * (e >> 1)]);
        }
        // ---- R0 of this warp's channels; before[nt][2 hh + e]: cumulative log-decay in front of token g + 8 hh of the block
        float sum[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};      // of the blocks so far (every row the same)
#pragma unroll
        for (int ks = 0; ks < kCB / 16; ++ks) {
            uint32_t wb[4];
            ldmatrix_x4_trans(wb[0], wb[1], wb[2], wb[3], sm.w[stage] + ks * 2048 + tile_row);
            if (kSplitHere) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int s = 16 * ks + 8 * (i & 1) + 2 * q;
                    wb[i] &= (s >= lo && s < hi ? 0xffffu : 0u) | (s + 1 >= lo && s + 1 < hi ? 0xffff0000u : 0u);
                }
            }
            uint32_t r0[4];           // in the order (hh, nt) = 00, 10, 01, 11
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                float before[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) before[e] = sum[nt][e];
                mma_bf16(before, earlier, kOnes, 0u, earlier, wb[2 * nt], wb[2 * nt + 1]);
                mma_bf16(sum[nt], kOnes, kOnes, kOnes, kOnes, wb[2 * nt], wb[2 * nt + 1]);
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int t = 16 * ks + g + 8 * hh;
                    uint32_t rw = *reinterpret_cast<const uint32_t*>(sm.r[stage] + ks * 2048 + (tile_word ^ (16 * nt)) + 1024 * hh);
                    if (kSplitHere && !(t >= lo && t < hi)) rw = 0;
                    const float2 rv = unpack2(rw);
                    r0[2 * nt + hh] = pack2(rv.x * exp_fast(before[2 * hh]), rv.y * exp_fast(before[2 * hh + 1]));
                }
            }
            if (starts != 0) {        // nothing from the first flag on sees the entering state
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const bool first = (starts & ((2ull << (16 * ks + g + 8 * hh)) - 1ull)) == 0;
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) r0[2 * nt + hh] = first ? r0[2 * nt + hh] : 0u;
                }
            }
            __syncwarp();             // (the block's rows of this warp's channels have been read)
            stmatrix_x4(sm.r[stage] + ks * 2048 + tile_row, r0[0], r0[1], r0[2], r0[3]);
        }
        if (g == 0) {
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
                *reinterpret_cast<float2*>(&sm.wc[j0 + 8 * nt + 2 * q]) = starts == 0 ? make_float2(exp_fast(sum[nt][0]), exp_fast(sum[nt][1])) : make_float2(0.f, 0.f);
        }
        __syncthreads();              // R0 and the step's decay are complete
        // dS0^T = dS_C^T diag(exp(c_C)) [no start in the step] + dY^T R0
#pragma unroll
        for (int np = 0; np < 4; ++np) {
            const float2 w0 = *reinterpret_cast<const float2*>(&sm.wc[16 * np + 2 * q]);
            const float2 w1 = *reinterpret_cast<const float2*>(&sm.wc[16 * np + 8 + 2 * q]);
            acc[2 * np][0] *= w0.x; acc[2 * np][1] *= w0.y; acc[2 * np][2] *= w0.x; acc[2 * np][3] *= w0.y;
            acc[2 * np + 1][0] *= w1.x; acc[2 * np + 1][1] *= w1.y; acc[2 * np + 1][2] *= w1.x; acc[2 * np + 1][3] *= w1.y;
        }
        if (has_dy) {
#pragma unroll
            for (int ks = 0; ks < kCB / 16; ++ks) {
                uint32_t y[4];
                ldmatrix_x4_trans(y[0], y[1], y[2], y[3], sm.dy[stage] + ks * 2048 + tile_row);
#pragma unroll
                for (int np = 0; np < 4; ++np) {
                    uint32_t b0, b1, b2, b3;
                    ldmatrix_x4_trans(b0, b1, b2, b3, sm.r[stage] + ks * 2048 + block_row(np));
                    mma_bf16(acc[2 * np], y[0], y[2], y[1], y[3], b0, b1);
                    mma_bf16(acc[2 * np + 1], y[0], y[2], y[1], y[3], b2, b3);
                }
            }
        }
    };
    for (int c = nB - 1; c >= c_stop - 1; --c) {
        // the state gradient behind the last step of a run (before anything of that step is applied), for the CTA of
        // the gradient kernel that walks the run
        if ((c + 1) % run_steps == 0 && c + 1 < nB) {
            bf* dst = dsck + ((size_t)bh * n_runs + c / run_steps) * kN * kN;
#pragma unroll
            for (int ni = 0; ni < 8; ++ni) {
                *reinterpret_cast<uint32_t*>(dst + (size_t)(j0 + g) * kN + 8 * ni + 2 * q) = pack2(acc[ni][0], acc[ni][1]);
                *reinterpret_cast<uint32_t*>(dst + (size_t)(j0 + g + 8) * kN + 8 * ni + 2 * q) = pack2(acc[ni][2], acc[ni][3]);
            }
        }
        if (c < c_stop) break;
        if (split && c == c_out) {
#pragma unroll 1
            for (int part = 1; part >= 0; --part) walk(std::true_type{}, c, part);
        } else {
            walk(std::false_type{}, c, 0);
        }
    }
    if (!waited && status != nullptr) atomicExch(status, 5);
}

// du of a (batch, head): the runs' shares added in a fixed order
__global__ void wkv6_reduce_runs_kernel(int BH, int n_runs, const float* partial, const int* __restrict__ residual_mark,
                                        float* __restrict__ du_head) {
    let_next_in();
    if (word_behind(residual_mark) != 0) return;
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= BH * kN) return;
    const int bh = idx / kN, i = idx % kN;
    float sum = 0.f;
    for (int rho = 0; rho < n_runs; ++rho) sum += partial[((size_t)bh * n_runs + rho) * kN + i];
    du_head[idx] = sum;
}

}  // namespace

// How the backward cuts a sequence: runs of 16 chunks (256 tokens) once there are at least two of them.
constexpr int kRunLen = kRunLen6;
static int runs_of(int T) {
    const int nC = (T + kC6 - 1) / kC6;
    return nC >= 2 * kRunLen ? (nC + kRunLen - 1) / kRunLen : 1;
}
struct Layout6 {
    size_t states, scores, dsck, partial, end;
};
static Layout6 layout6(int B, int T, int H) {
    const size_t nC = (size_t)(T + kC6 - 1) / kC6, runs = (size_t)runs_of(T), tile = (size_t)kN * kN * sizeof(bf);
    Layout6 l;
    l.states = 0;                                              // every chunk's entering state, and the second part of a split one
    l.scores = l.states + (size_t)B * H * (nC + 1) * tile;     // its score block A^T (512 bytes)
    l.dsck = l.scores + (size_t)B * H * (nC + 1) * 32 * sizeof(uint4);   // the state gradient at the end of every run (written by the backward)
    l.partial = l.dsck + (size_t)B * H * runs * tile;          // the runs' shares of du (fp32)
    l.end = l.partial + (size_t)B * H * runs * kN * sizeof(float);
    return l;
}

size_t wkv6_chunk_residual_bytes(int B, int T, int H) { return layout6(B, T, H).end; }

int wkv6_chunk_fwd(cudaStream_t st, int B, int T, int H, const void* r, const void* k, const void* v, const void* w,
                   int per_token, const void* u, const void* s0, const uint32_t* length, const uint8_t* ns, void* y,
                   void* s_out, void* residual, int* residual_mark, int** flag, int* ticket) {
    static DeviceOnce smem_attr;
    if (!smem_attr.ok([]() { return cudaFuncSetAttribute(wkv6_chunk_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Fwd6cSmem)); }))
        return B200WKV_ELAUNCH;
    *flag = wkv_call_flag(ticket);
    if (*flag == nullptr) return B200WKV_ELAUNCH;
    const void* streams[5] = {r, k, v, per_token ? w : nullptr, y};
    SeqMaps maps;
    if (!make_seq_maps(&maps, streams, 5, B, T, H, kC6)) return B200WKV_ELAUNCH;
    wkv6_chunk_fwd_kernel<<<B * H, 128, sizeof(Fwd6cSmem), st>>>(T, H, (const bf*)r, (const bf*)k, (const bf*)v, (const bf*)w, per_token,
                                                                (const bf*)u, (const bf*)s0, length, ns, (bf*)y, (bf*)s_out,
                                                                (bf*)residual,
                                                                residual != nullptr ? reinterpret_cast<uint4*>(static_cast<char*>(residual) + layout6(B, T, H).scores) : nullptr, *flag, *ticket, residual_mark, maps);
    return cudaGetLastError() == cudaSuccess ? B200WKV_OK : B200WKV_ELAUNCH;
}

int wkv6_chunk_bwd(cudaStream_t st, int B, int T, int H, const void* r, const void* k, const void* v, const void* w,
                   const void* u, const uint32_t* length, const uint8_t* ns, const void* dy, const void* ds_out,
                   void* residual, const int* residual_mark, void* dr, void* dk, void* dv, void* dw, void* du, void* ds0) {
    static DeviceOnce smem_attr;
    if (!smem_attr.ok([]() {
            cudaError_t e = cudaFuncSetAttribute(wkv6_chunk_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Bwd6cSmem));
            if (e != cudaSuccess) return e;
            return cudaFuncSetAttribute(wkv6_carry_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Carry6Smem));
        }))
        return B200WKV_ELAUNCH;
    const Layout6 lay = layout6(B, T, H);
    char* base = static_cast<char*>(residual);
    const int n_runs = runs_of(T);
    bf* dsck = reinterpret_cast<bf*>(base + lay.dsck);
    float* partial = reinterpret_cast<float*>(base + lay.partial);
    if (n_runs > 1) {
        const void* streams[3] = {r, w, dy};
        SeqMaps maps;
        if (!make_seq_maps(&maps, streams, 3, B, T, H, kCB)) return B200WKV_ELAUNCH;
        wkv6_carry_bwd_kernel<<<B * H, 128, sizeof(Carry6Smem), st>>>(T, H, (const bf*)r, length, ns, dy != nullptr ? 1 : 0, (const bf*)ds_out,
                                                                     residual_mark, n_runs, kRunLen, dsck, wkv7_chunk_status_word(), maps);
        if (cudaGetLastError() != cudaSuccess) return B200WKV_ELAUNCH;
    }
    const void* streams[9] = {r, k, v, w, dy, dr, dk, dv, dw};
    SeqMaps maps;
    if (!make_seq_maps(&maps, streams, 9, B, T, H, kC6)) return B200WKV_ELAUNCH;
    // (behind the carry, where there is one)
    if (launch_in_chain(n_runs == 1, wkv6_chunk_bwd_kernel, B * H * n_runs, 128, sizeof(Bwd6cSmem), st, T, H, (const bf*)u, length, ns, dy != nullptr ? 1 : 0,
                        (const bf*)ds_out, (const bf*)(base + lay.states), (const uint4*)(base + lay.scores), residual_mark, (bf*)dr, (bf*)dk, (bf*)dv,
                        (bf*)dw, (float*)du, (bf*)ds0, n_runs, n_runs > 1 ? kRunLen : (T + kC6 - 1) / kC6, dsck, partial, wkv7_chunk_status_word(),
                        maps) != cudaSuccess)
        return B200WKV_ELAUNCH;
    if (n_runs > 1) {
        const int total = B * H * kN;
        if (launch_behind(wkv6_reduce_runs_kernel, (total + 255) / 256, 256, 0, st, B * H, n_runs, partial, residual_mark, (float*)du) != cudaSuccess)
            return B200WKV_ELAUNCH;
    }
    return B200WKV_OK;
}

}  // namespace b200wkv
