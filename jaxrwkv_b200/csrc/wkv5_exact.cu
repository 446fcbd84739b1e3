// RWKV-5 / 5.2 (one constant decay per key channel), bf16 streams: fp32-accurate matrix products in runs of 64 tokens that are
// walked side by side.
//
// The gradient of a constant decay is a sum over ALL tokens of terms that largely cancel, so training calls keep
// fp32 accuracy throughout, and so do the host path's calls without gradients, whose results are the same bits.  Token by token on CUDA cores (wkv6_seq.cu) that costs 0.5 us per token and head forward and
// 1.1 us backward on a chain as long as the sequence.  Here a chunk of 16 tokens is a handful of matrix products on
// mma.sync m16n8k8 tf32 tiles; every fp32 factor goes in as two tf32 numbers (x = hi + lo, 22 bits), products of two such
// factors as hi hi + hi lo + lo hi; bf16 values are exact in tf32.  With d = the decay, t, s local to the chunk, m = 8:
//     R0_t = r_t d^t    R~_t = r_t d^{t-1-m}    K~_s = k_s d^{m-s}    K^_s = k_s d^{n-1-s}
//     A_ts = R~_t . K~_s (s < t), A_tt = sum r u k;   Y = R0 S + A V;   S' = d^n S + K^^T V
// and, with dS the gradient of S' and dA = dY V^T (s < t):
//     dr = d^t (dY S^T) + d^{t-1-m} (dA K~) + u k (dy.v)      dk = d^{n-1-s} (V dS^T) + d^{m-s} (dA^T R~) + u r (dy.v)
//     dv = K^ dS + A^T dY                                     dS_before = d^n dS + R0^T dY
//     d * dd = sum over all factors of (exponent) x (factor . its gradient)
// A start flag masks A, the rows of R0 / K^ and the carried state (wkv6_chunk.cu).  A `length` inside a chunk: the
// forward walks the chunk in two parts, the backward adds the returned state's cotangent as a second dS that ends there.
//
// Time is cut into runs of four chunks.  Forward: (1) every run reduces its tokens to the state they leave from zero;
// (2) an elementwise scan over the runs turns those into entering states; (3) every run walks its chunks from there,
// writing y and the state entering each chunk, in the format of wkv6_seq.cu (fp32, every 16 tokens): the two families
// are interchangeable per head.  Backward: the same three steps in reverse; the state gradients between runs lie in the
// rows of dr and dk of the run in front, which that run reads before it writes them.
//
// Measured at B=4, T=1024, H=32: forward 515 -> 24 + 9 + 80 us, backward 1127 -> 30 + 9 + 194 + 3 us.  The outputs and the
// gradients use the shared-memory path to 78 and 76 % of its peak and 48 and 43 % of the issue slots; the gradient kernel's
// warps wait longest for the checkpoint's rows out of global memory (1.3 cycles per issued instruction), then for shared memory (1.1).
// A 64-term product of a split fp32 factor with a bf16 row has a relative error of 1.3e-7 (an fp32 fma chain 1.5e-7), of two
// split factors 3.5e-7; results are rounded to bf16, 1.7e-3.
// Powers of d outside d^{+-8} fp32 range: a head with a channel outside [1e-4, 1] is left to wkv6_seq.cu.
#include <initializer_list>
#include "common.cuh"
#include "device_once.cuh"

namespace b200wkv {
namespace {

typedef __nv_bfloat16 bf;
constexpr int kC = 16, kRunChunks = 4, kRun = kC * kRunChunks;
constexpr int kMid = 8;
constexpr int kPitch = 72;       // of row tiles read along the row: 8-byte fragment reads of 4 rows fill the 32 banks
constexpr int kPitchT = 68;      // of tiles read down the columns: rows two apart are 8 banks apart
constexpr int kPow = 17;         // d^0 .. d^16
constexpr int kNeg = 8;          // d^-1 .. d^-8

__device__ __forceinline__ bool in_domain(const bf* w_head) {   // of the whole head; all threads of the CTA call it
    const int i = threadIdx.x & 63;
    const float d = __bfloat162float(w_head[i]);
    return __syncthreads_and(d >= 1e-4f && d <= 1.f) != 0;
}

// What is not a number ends at a start flag in the token-sequential kernels, but 0 x NaN would carry it on here.  A chunk with
// flags that meets any in what the masks' zeros are multiplied with sets its head's word, and the head is left to wkv6_seq.cu.
__device__ __forceinline__ bool odd(uint32_t two) { return (two & 0x7f80u) == 0x7f80u || (two & 0x7f800000u) == 0x7f800000u; }   // bf16
__device__ __forceinline__ bool odd_rows(const bf* tile_at) {          // 8 elements
    const uint4 x = *reinterpret_cast<const uint4*>(tile_at);
    return odd(x.x) || odd(x.y) || odd(x.z) || odd(x.w);
}
__device__ __forceinline__ bool odd_tiles(const float (*acc)[4]) {
    float z = 0.f;
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) z = fmaf(acc[n][e], 0.f, z);
    return z != 0.f;
}

struct Pow {
    float p[kPow][kN], n[kNeg + 1][kN];    // d^e, d^-e
    __device__ __forceinline__ float at(int e, int i) const { return e >= 0 ? p[e][i] : n[-e][i]; }
};
// Each power to the last bit: carried as an unevaluated sum hi + lo (the exact product by fma), threads 0-63 upwards, 64-127
// down.  (In fp64 this prologue was a fifth of the kernels' time.)
__device__ __forceinline__ void fill_powers(Pow& pw, const bf* w_head) {
    const int i = threadIdx.x & 63;
    const float d = __bfloat162float(w_head[i]);
    float hi = 1.f, lo = 0.f;
    if (threadIdx.x < kN) {
#pragma unroll
        for (int e = 0; e < kPow; ++e) {
            pw.p[e][i] = hi + lo;
            const float h = hi * d;
            lo = fmaf(lo, d, fmaf(hi, d, -h));
            hi = h;
        }
    } else {
        const float ih = 1.f / d, il = fmaf(-d, ih, 1.f) * ih;
#pragma unroll
        for (int e = 0; e <= kNeg; ++e) {
            pw.n[e][i] = hi + lo;
            const float h = hi * ih;
            lo = fmaf(lo, ih, fmaf(hi, il, fmaf(hi, ih, -h)));
            hi = h;
        }
    }
}

// fp32 as two tf32 numbers: the hardware reads the upper 19 bits
struct Split {
    uint32_t hi, lo;
    __device__ __forceinline__ Split() {}
    __device__ __forceinline__ explicit Split(float x) {
        hi = __float_as_uint(x) & 0xffffe000u;
        lo = __float_as_uint(x - __uint_as_float(hi));
    }
};
struct A2 { Split a[4]; };       // left operand 16x8: rows g, g + 8; the k index t of a lane stands for columns 2t, 2t + 1
struct B2 { Split b[2]; };       // right operand 8x8
struct A1 { uint32_t a[4]; };    // the same, exact in tf32
struct B1 { uint32_t b[2]; };

__device__ __forceinline__ void mma(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma(float* c, const A2& a, const B2& b) {
    mma(c, a.a[0].lo, a.a[1].lo, a.a[2].lo, a.a[3].lo, b.b[0].hi, b.b[1].hi);
    mma(c, a.a[0].hi, a.a[1].hi, a.a[2].hi, a.a[3].hi, b.b[0].lo, b.b[1].lo);
    mma(c, a.a[0].hi, a.a[1].hi, a.a[2].hi, a.a[3].hi, b.b[0].hi, b.b[1].hi);
}
__device__ __forceinline__ void mma(float* c, const A2& a, const B1& b) {
    mma(c, a.a[0].lo, a.a[1].lo, a.a[2].lo, a.a[3].lo, b.b[0], b.b[1]);
    mma(c, a.a[0].hi, a.a[1].hi, a.a[2].hi, a.a[3].hi, b.b[0], b.b[1]);
}
__device__ __forceinline__ void mma(float* c, const A1& a, const B2& b) {
    mma(c, a.a[0], a.a[1], a.a[2], a.a[3], b.b[0].lo, b.b[1].lo);
    mma(c, a.a[0], a.a[1], a.a[2], a.a[3], b.b[0].hi, b.b[1].hi);
}
__device__ __forceinline__ void mma(float* c, const A1& a, const B1& b) { mma(c, a.a[0], a.a[1], a.a[2], a.a[3], b.b[0], b.b[1]); }

// An accumulator tile (rows g, g + 8; columns 2t, 2t + 1) as a left operand, and as a right operand whose n index is the
// tile's row (upper half: rows 0-7) and whose k index is its column.
__device__ __forceinline__ A2 as_left(const float* c) {
    A2 x;
    x.a[0] = Split(c[0]); x.a[1] = Split(c[2]); x.a[2] = Split(c[1]); x.a[3] = Split(c[3]);
    return x;
}
__device__ __forceinline__ B2 as_right(const float* c, int half) {
    B2 x;
    x.b[0] = Split(c[2 * half]); x.b[1] = Split(c[2 * half + 1]);
    return x;
}
// fragments of fp32 row tiles [row][column]: left / right operand with k along the row
__device__ __forceinline__ A2 rows_left(const float* tile, int pitch, int ks, int g, int q) {
    const float2 u = *reinterpret_cast<const float2*>(tile + g * pitch + 8 * ks + 2 * q);
    const float2 d = *reinterpret_cast<const float2*>(tile + (g + 8) * pitch + 8 * ks + 2 * q);
    A2 x;
    x.a[0] = Split(u.x); x.a[1] = Split(d.x); x.a[2] = Split(u.y); x.a[3] = Split(d.y);
    return x;
}
__device__ __forceinline__ B2 rows_right(const float* tile, int pitch, int nt, int ks, int g, int q) {
    const float2 u = *reinterpret_cast<const float2*>(tile + (8 * nt + g) * pitch + 8 * ks + 2 * q);
    B2 x;
    x.b[0] = Split(u.x); x.b[1] = Split(u.y);
    return x;
}
// the same with k down the columns: element (k, n) of `tile`, n from column c0
__device__ __forceinline__ A2 cols_left(const float* tile, int pitch, int ks, int c0, int g, int q) {
    const float* p = tile + (8 * ks + 2 * q) * pitch + c0 + g;
    A2 x;
    x.a[0] = Split(p[0]); x.a[1] = Split(p[8]); x.a[2] = Split(p[pitch]); x.a[3] = Split(p[pitch + 8]);
    return x;
}
__device__ __forceinline__ B2 cols_right(const float* tile, int pitch, int ks, int c0, int g, int q) {
    const float* p = tile + (8 * ks + 2 * q) * pitch + c0 + g;
    B2 x;
    x.b[0] = Split(p[0]); x.b[1] = Split(p[pitch]);
    return x;
}
// bf16 tiles [token][channel] of kPitch elements: exact
__device__ __forceinline__ uint32_t low(uint32_t two) { return two << 16; }
__device__ __forceinline__ uint32_t high(uint32_t two) { return two & 0xffff0000u; }
__device__ __forceinline__ uint32_t one(const bf* p) { return (uint32_t)*reinterpret_cast<const unsigned short*>(p) << 16; }
__device__ __forceinline__ A1 raw_rows_left(const bf* tile, int ks, int g, int q) {
    const uint32_t u = *reinterpret_cast<const uint32_t*>(tile + g * kPitch + 8 * ks + 2 * q);
    const uint32_t d = *reinterpret_cast<const uint32_t*>(tile + (g + 8) * kPitch + 8 * ks + 2 * q);
    return A1{{low(u), low(d), high(u), high(d)}};
}
__device__ __forceinline__ B1 raw_rows_right(const bf* tile, int nt, int ks, int g, int q) {
    const uint32_t u = *reinterpret_cast<const uint32_t*>(tile + (8 * nt + g) * kPitch + 8 * ks + 2 * q);
    return B1{{low(u), high(u)}};
}
__device__ __forceinline__ A1 raw_cols_left(const bf* tile, int ks, int c0, int g, int q) {
    const bf* p = tile + (8 * ks + 2 * q) * kPitch + c0 + g;
    return A1{{one(p), one(p + 8), one(p + kPitch), one(p + kPitch + 8)}};
}
__device__ __forceinline__ B1 raw_cols_right(const bf* tile, int ks, int c0, int g, int q) {
    const bf* p = tile + (8 * ks + 2 * q) * kPitch + c0 + g;
    return B1{{one(p), one(p + kPitch)}};
}

// bits lo .. hi - 1
__device__ __forceinline__ uint32_t bits(int lo, int hi) { return ((1u << hi) - 1u) & ~((1u << lo) - 1u); }

// A chunk's rows of one stream on their way to shared memory, rows behind the end as zeros; 128 threads, a 16-byte piece each
struct Ahead {
    uint4 x;
    __device__ __forceinline__ void fetch(const bf* src, size_t base, size_t stride, int t0, int Tlen) {
        const int t = t0 + (threadIdx.x >> 3);
        x = make_uint4(0u, 0u, 0u, 0u);
        if (src != nullptr && t >= 0 && t < Tlen) x = *reinterpret_cast<const uint4*>(src + base + (size_t)t * stride + (threadIdx.x & 7) * 8);
    }
    __device__ __forceinline__ void put(bf (*tile)[kPitch]) const { *reinterpret_cast<uint4*>(&tile[threadIdx.x >> 3][(threadIdx.x & 7) * 8]) = x; }
};
// Products over all 64 channels whose 16 x 16 result every warp needs: each warp takes a quarter of the channels, and the
// quarters are added through shared memory.
struct Quarters {
    float4 q[4][2][32];
    __device__ __forceinline__ void put(int warp, int lane, const float (*c)[4]) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) q[warp][nt][lane] = make_float4(c[nt][0], c[nt][1], c[nt][2], c[nt][3]);
    }
    __device__ __forceinline__ void sum(int lane, float (*c)[4]) const {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            const float4 a = q[0][nt][lane], b = q[1][nt][lane], d = q[2][nt][lane], e = q[3][nt][lane];
            c[nt][0] = (a.x + b.x) + (d.x + e.x); c[nt][1] = (a.y + b.y) + (d.y + e.y);
            c[nt][2] = (a.z + b.z) + (d.z + e.z); c[nt][3] = (a.w + b.w) + (d.w + e.w);
        }
    }
};
// start flags of the run's chunks, one bit per token
__device__ __forceinline__ void load_starts(uint32_t* masks, const uint8_t* ns, int t0, int Tlen) {
    const int t = t0 + threadIdx.x;
    const unsigned m = __ballot_sync(0xffffffffu, threadIdx.x < kRun && t < Tlen && ns[t] != 0);
    if (threadIdx.x < kRun && (threadIdx.x & 31) == 0) {
        masks[threadIdx.x >> 4] = m & 0xffffu;
        masks[(threadIdx.x >> 4) + 1] = m >> 16;
    }
}

// ------------------------------------------------------------------ forward ---------
struct FwdSmem5 {
    bf r[kC][kPitch], k[kC][kPitch], v[kC][kPitch];
    Quarters scores;
    float rt[kC][kPitch], kt[kC][kPitch], r0[kC][kPitch], kh[kC][kPitchT];
    bf ys[kC][kPitch];
    float diag[kC];              // sum_i r u k
    Pow pw;
    uint32_t starts[kRunChunks];
};

// `states`: n_states fp32 states per head, per_run of them per run, the first of which is the one entering the run.  A call whose
// residual they are keeps one per chunk (per_run = kRunChunks: the checkpoints), a call without a residual one per run.
// kOutputs false: the state that the run's tokens leave from zero, into the slot of the run behind (no CTA for
// the last run).  True: y, the checkpoints of the run's chunks behind the first, and the returned state.
// 128 threads; warp w holds the rows j = 16 w .. of S^T[j][i] as accumulator tiles.
template <bool kOutputs>
__global__ void __launch_bounds__(128, 4)
wkv5_fwd_kernel(int Tlen, int H, int runs, int n_states, int per_run, const bf* __restrict__ r, const bf* __restrict__ k, const bf* __restrict__ v,
                const bf* __restrict__ w, const bf* __restrict__ u, const bf* __restrict__ s0, const uint32_t* __restrict__ length,
                const uint8_t* __restrict__ new_starts, bf* __restrict__ y, bf* __restrict__ s_out, float* states,
                int* __restrict__ odd_heads, int* __restrict__ residual_mark) {
    let_next_in();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FwdSmem5& sm = *reinterpret_cast<FwdSmem5*>(smem_raw);
    const int bh = blockIdx.x / runs, run = blockIdx.x % runs, bi = bh / H, h = bh % H;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3, j0 = 16 * warp;
    if (kOutputs && residual_mark != nullptr && blockIdx.x == 0 && tid == 0) *residual_mark = 1;   // fp32 checkpoints
    if (!in_domain(w + (size_t)h * kN)) {
        wait_for_grid_in_front();
        return;
    }
    const size_t stride = (size_t)H * kN, base = (size_t)bi * Tlen * stride + (size_t)h * kN;
    const int t_run = run * kRun, L = min((int)length[bi], Tlen);
    float* const slots = states + (size_t)bh * n_states * kN * kN;
    float acc[8][4];             // acc[ni][e] = S[i = 8 ni + 2 q + (e & 1)][j = j0 + g + 8 (e >> 1)]
    auto element = [&](int ni, int e) { return (8 * ni + 2 * q + (e & 1)) * kN + j0 + g + 8 * (e >> 1); };
    Ahead r_next, k_next, v_next;
    auto fetch = [&](int t0) {
        if (kOutputs) r_next.fetch(r, base, stride, t0, Tlen);
        k_next.fetch(k, base, stride, t0, Tlen);
        v_next.fetch(v, base, stride, t0, Tlen);
    };
    fetch(t_run);
    load_starts(sm.starts, new_starts + (size_t)bi * Tlen, t_run, Tlen);
    fill_powers(sm.pw, w + (size_t)h * kN);
    wait_for_grid_in_front();    // (what is above depends on the operands alone)
    if (kOutputs) {
        const float* from = slots + (size_t)run * per_run * kN * kN;
#pragma unroll
        for (int ni = 0; ni < 8; ++ni)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[ni][e] = from[element(ni, e)];
    } else {
#pragma unroll
        for (int ni = 0; ni < 8; ++ni)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[ni][e] = 0.f;
    }
    auto write_state = [&](bf* to) {
#pragma unroll
        for (int ni = 0; ni < 8; ++ni)
#pragma unroll
            for (int e = 0; e < 4; ++e) to[(size_t)bh * kN * kN + element(ni, e)] = __float2bfloat16_rn(acc[ni][e]);
    };
    if (kOutputs && run == 0 && L == 0) {       // the input state comes back as it was given
        for (int i = tid; i < kN * kN / 8; i += 128)
            reinterpret_cast<uint4*>(s_out + (size_t)bh * kN * kN)[i] = reinterpret_cast<const uint4*>(s0 + (size_t)bh * kN * kN)[i];
    }
    // operand tiles: channels cp, cp + 1 of the tokens 4 qt .. 4 qt + 3
    const int cp = lane * 2, qt = warp;
    const float2 uu = kOutputs ? make_float2(__bfloat162float(u[(size_t)h * kN + cp]), __bfloat162float(u[(size_t)h * kN + cp + 1])) : make_float2(0.f, 0.f);
    __syncthreads();

    for (int c = 0; c < kRunChunks; ++c) {
        const int t0 = t_run + c * kC, n_chunk = min(kC, Tlen - t0);
        if (n_chunk <= 0) break;
        const bf(*rr)[kPitch] = sm.r;
        const bf(*kk)[kPitch] = sm.k;
        const bf* vv = &sm.v[0][0];
        if (kOutputs) r_next.put(sm.r);
        k_next.put(sm.k);
        v_next.put(sm.v);
        __syncthreads();
        if (c + 1 < kRunChunks) fetch(t0 + kC);
        const uint32_t starts = sm.starts[c];
        if (kOutputs && starts != 0 && (odd_tiles(acc) || odd_rows(&sm.v[tid >> 3][(tid & 7) * 8]))) odd_heads[bh] = 1;
        if (kOutputs && c > 0 && per_run == kRunChunks) {
            float* to = slots + (size_t)(run * kRunChunks + c) * kN * kN;
#pragma unroll
            for (int ni = 0; ni < 8; ++ni)
#pragma unroll
                for (int e = 0; e < 4; ++e) to[element(ni, e)] = acc[ni][e];
        }
        // the chunk in one part, or in two around the token whose state is returned
        for (int lo = 0, hi; lo < n_chunk; lo = hi) {
            hi = kOutputs && L > t0 + lo && L < t0 + n_chunk ? L - t0 : n_chunk;
            float dsum[4];
#pragma unroll
            for (int tt = 0; tt < 4; ++tt) {
                const int t = 4 * qt + tt;
                const bool in = t >= lo && t < hi, first = in && (starts & bits(lo, t + 1)) == 0, last = in && (starts & bits(t + 1, hi)) == 0;
                const uint32_t k2 = *reinterpret_cast<const uint32_t*>(&kk[t][cp]);
                const float2 kf = make_float2(__uint_as_float(low(k2)), __uint_as_float(high(k2)));
                const int e_hat = last ? hi - 1 - t : 0;
                const float2 ph = *reinterpret_cast<const float2*>(&sm.pw.p[e_hat][cp]);
                *reinterpret_cast<float2*>(&sm.kh[t][cp]) = last ? make_float2(kf.x * ph.x, kf.y * ph.y) : make_float2(0.f, 0.f);
                if (kOutputs) {
                    const uint32_t r2 = *reinterpret_cast<const uint32_t*>(&rr[t][cp]);
                    const float2 rf = make_float2(__uint_as_float(low(r2)), __uint_as_float(high(r2)));
                    const float2 p0 = *reinterpret_cast<const float2*>(&sm.pw.p[first ? t - lo : 0][cp]);
                    const int em = t - 1 - kMid;
                    *reinterpret_cast<float2*>(&sm.r0[t][cp]) = first ? make_float2(rf.x * p0.x, rf.y * p0.y) : make_float2(0.f, 0.f);
                    *reinterpret_cast<float2*>(&sm.rt[t][cp]) =
                        t == 0 ? make_float2(0.f, 0.f) : make_float2(rf.x * sm.pw.at(em, cp), rf.y * sm.pw.at(em, cp + 1));
                    *reinterpret_cast<float2*>(&sm.kt[t][cp]) = make_float2(kf.x * sm.pw.at(kMid - t, cp), kf.y * sm.pw.at(kMid - t, cp + 1));
                    dsum[tt] = rf.x * uu.x * kf.x + rf.y * uu.y * kf.y;
                }
            }
            if (kOutputs) {
#pragma unroll
                for (int tt = 0; tt < 4; ++tt) {
#pragma unroll
                    for (int m = 1; m < 32; m <<= 1) dsum[tt] += __shfl_xor_sync(0xffffffffu, dsum[tt], m);
                    if (lane == 0) sm.diag[4 * qt + tt] = dsum[tt];
                }
            }
            __syncthreads();
            if (kOutputs) {
                float yacc[2][4], sc[2][4];      // Y^T: rows j, columns t; A: rows t, columns s
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int e = 0; e < 4; ++e) yacc[nt][e] = sc[nt][e] = 0.f;
#pragma unroll
                for (int kq = 0; kq < 2; ++kq) {
                    const A2 ra = rows_left(&sm.rt[0][0], kPitch, 2 * warp + kq, g, q);
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) mma(sc[nt], ra, rows_right(&sm.kt[0][0], kPitch, nt, 2 * warp + kq, g, q));
                }
                sm.scores.put(warp, lane, sc);
#pragma unroll
                for (int ks = 0; ks < 8; ++ks) {
                    const A2 sa = as_left(acc[ks]);
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) mma(yacc[nt], sa, rows_right(&sm.r0[0][0], kPitch, nt, ks, g, q));
                }
                __syncthreads();
                sm.scores.sum(lane, sc);
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int t = g + 8 * (e >> 1), s = 8 * nt + 2 * q + (e & 1);
                        const bool pair = s >= lo && s < t && t < hi && (starts & bits(s + 1, t + 1)) == 0;
                        const bool diag = s == t && t >= lo && t < hi;
                        sc[nt][e] = pair ? sc[nt][e] : diag ? sm.diag[t] : 0.f;
                    }
#pragma unroll
                for (int kt = 0; kt < 2; ++kt) {
                    const A1 va = raw_cols_left(vv, kt, j0, g, q);
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) mma(yacc[nt], va, as_right(sc[kt], nt));
                }
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int t = 8 * nt + 2 * q + (e & 1);
                        if (t >= lo && t < hi) sm.ys[t][j0 + g + 8 * (e >> 1)] = __float2bfloat16_rn(yacc[nt][e]);
                    }
            }
            const bool keep = (starts & bits(lo, hi)) == 0;
#pragma unroll
            for (int ni = 0; ni < 8; ++ni) {
                const float2 d = *reinterpret_cast<const float2*>(&sm.pw.p[hi - lo][8 * ni + 2 * q]);
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[ni][e] = keep ? acc[ni][e] * ((e & 1) ? d.y : d.x) : 0.f;
            }
#pragma unroll
            for (int kt = 0; kt < 2; ++kt) {
                const A1 va = raw_cols_left(vv, kt, j0, g, q);
#pragma unroll
                for (int ni = 0; ni < 8; ++ni) mma(acc[ni], va, cols_right(&sm.kh[0][0], kPitchT, kt, 8 * ni, g, q));
            }
            if (kOutputs && t0 + hi == L) write_state(s_out);
            __syncthreads();     // the tiles have been read
        }
        if (kOutputs) {
            const int row = tid >> 3, piece = (tid & 7) * 8;
            if (row < n_chunk)
                *reinterpret_cast<uint4*>(y + base + (size_t)(t0 + row) * stride + piece) = *reinterpret_cast<const uint4*>(&sm.ys[row][piece]);
            // (barriers of the next chunk lie between these reads and the next writes of ys)
        }
    }
    if (!kOutputs) {
        float* to = slots + (size_t)(run + 1) * per_run * kN * kN;
#pragma unroll
        for (int ni = 0; ni < 8; ++ni)
#pragma unroll
            for (int e = 0; e < 4; ++e) to[element(ni, e)] = acc[ni][e];
    }
}

// The scan over the runs of one head: slot(next) = keep d^64 slot(this) + slot(next), for `steps` steps.  Forward: this =
// the state entering a run (the first from s0), slots in `states`.  Backward (kForward false): from the last run but
// one down, slots in the rows of dr and dk (see run_slot()).  Four elements of a row per thread.
__device__ __forceinline__ float* run_slot(bf* dr, bf* dk, size_t base, size_t stride, int run, int i, int j) {
    return reinterpret_cast<float*>((j < 32 ? dr : dk) + base + (size_t)(run * kRun + i) * stride) + (j & 31);
}
template <bool kForward>
__global__ void __launch_bounds__(256)
wkv5_scan_kernel(int Tlen, int H, int runs, int n_states, int per_run, const bf* __restrict__ w, const bf* __restrict__ s0,
                 const uint8_t* __restrict__ new_starts, float* states, int* __restrict__ odd_heads, bf* dr, bf* dk) {
    extern __shared__ unsigned char keep[];      // per run: no start flag inside
    const int bh = blockIdx.x, bi = bh / H, h = bh % H, tid = threadIdx.x;
    let_next_in();
    if (kForward && blockIdx.y == 0 && tid == 0) odd_heads[bh] = 0;
    if (!in_domain(w + (size_t)h * kN)) {
        wait_for_grid_in_front();
        return;
    }
    for (int rn = tid >> 5; rn < runs; rn += 8) {
        const int t = rn * kRun + (tid & 31);
        const uint8_t* ns = new_starts + (size_t)bi * Tlen;
        const bool any = (t < Tlen && ns[t] != 0) || (t + 32 < Tlen && ns[t + 32] != 0);
        const unsigned m = __ballot_sync(0xffffffffu, any);
        if ((tid & 31) == 0) keep[rn] = m == 0;
    }
    __syncthreads();
    const int at = (blockIdx.y * 256 + tid) * 4, i = at / kN, j = at % kN;
    double d = (double)__bfloat162float(w[(size_t)h * kN + i]);
#pragma unroll
    for (int e = 1; e < kRun; e *= 2) d *= d;
    const float dn = (float)d;
    wait_for_grid_in_front();
    const size_t stride = (size_t)H * kN, base = (size_t)bi * Tlen * stride + (size_t)h * kN;
    auto slot = [&](int rn) {
        return reinterpret_cast<float4*>(kForward ? states + ((size_t)bh * n_states + (size_t)rn * per_run) * kN * kN + at
                                                  : run_slot(dr, dk, base, stride, rn, i, j));
    };
    auto step = [&](float4& x, const float4& add, int rn) {
        const float f = keep[rn] ? dn : 0.f;
        x = keep[rn] ? make_float4(fmaf(f, x.x, add.x), fmaf(f, x.y, add.y), fmaf(f, x.z, add.z), fmaf(f, x.w, add.w)) : add;
    };
    float4 x;
    if (kForward) {
        x = load4(s0 + (size_t)bh * kN * kN + at);
        *slot(0) = x;
        for (int rn = 0; rn + 1 < runs; rn += 4) {           // four slots in flight
            float4 a[4];
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if (rn + m + 1 < runs) a[m] = *slot(rn + m + 1);
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if (rn + m + 1 < runs) {
                    step(x, a[m], rn + m);
                    *slot(rn + m + 1) = x;
                }
        }
    } else {
        x = *slot(runs - 2);
        for (int rn = runs - 2; rn > 0; rn -= 4) {           // through run rn, into the slot of run rn - 1
            float4 a[4];
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if (rn - m > 0) a[m] = *slot(rn - m - 1);
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if (rn - m > 0) {
                    step(x, a[m], rn - m);
                    *slot(rn - m - 1) = x;
                }
        }
    }
}

// ------------------------------------------------------------------ backward --------
struct BwdSmem5 {
    bf r[kC][kPitch], k[kC][kPitch], v[kC][kPitch], dy[kC][kPitch];
    float rt[kC][kPitch], kt[kC][kPitch], r0[kC][kPitchT], kh[kC][kPitch];
    float ds[kN][kPitchT];       // the state gradient at hand, [key i][value j]
    union {
        Quarters sums[3];        // dA, dA^T, A^T
        bf out[3][kC][kPitch];   // dr, dk, dv
    };
    float dyv[kC], ruk[kC];
    Pow pw;
    uint32_t starts[kRunChunks];
};

// kGrads false: what the run's tokens (and the returned state's cotangent, where it enters inside) contribute to the state
// gradient in front of the run, into the slot of the run in front (no CTA for run 0).  True: all gradients of the run.
// Warp w holds the rows i = 16 w .. of dS[i][j] as accumulator tiles and, of dv, the columns j = 16 w ...
// part: [B H runs][2][64]: the run's shares of dw and du.
template <bool kGrads>
__global__ void __launch_bounds__(128, 3)
wkv5_bwd_kernel(int Tlen, int H, int runs, const bf* __restrict__ r, const bf* __restrict__ k, const bf* __restrict__ v,
                const bf* __restrict__ w, const bf* __restrict__ u, const uint32_t* __restrict__ length,
                const uint8_t* __restrict__ new_starts, const bf* __restrict__ dy, const bf* __restrict__ ds_out,
                const float* __restrict__ ckpt, int* __restrict__ odd_heads, bf* dr, bf* dk, bf* __restrict__ dv, float* __restrict__ part,
                bf* __restrict__ ds0) {
    let_next_in();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BwdSmem5& sm = *reinterpret_cast<BwdSmem5*>(smem_raw);
    const int n_here = kGrads ? runs : runs - 1;
    const int bh = blockIdx.x / n_here, run = blockIdx.x % n_here + (kGrads ? 0 : 1), bi = bh / H, h = bh % H;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3, i0 = 16 * warp;
    if (!in_domain(w + (size_t)h * kN)) {
        wait_for_grid_in_front();
        return;
    }
    const size_t stride = (size_t)H * kN, base = (size_t)bi * Tlen * stride + (size_t)h * kN;
    const int t_run = run * kRun, nC = (Tlen + kC - 1) / kC, L = min((int)length[bi], Tlen);
    float acc[8][4];             // acc[nj][e] = dS[i = i0 + g + 8 (e >> 1)][j = 8 nj + 2 q + (e & 1)]
    const int row_u = i0 + g, row_d = i0 + g + 8;
    Ahead r_next, k_next, v_next, dy_next;
    auto fetch = [&](int t0) {
        r_next.fetch(r, base, stride, t0, Tlen);
        dy_next.fetch(dy, base, stride, t0, Tlen);
        if (kGrads) {
            k_next.fetch(k, base, stride, t0, Tlen);
            v_next.fetch(v, base, stride, t0, Tlen);
        }
    };
    fetch(t_run + (kRunChunks - 1) * kC);
    load_starts(sm.starts, new_starts + (size_t)bi * Tlen, t_run, Tlen);
    fill_powers(sm.pw, w + (size_t)h * kN);
    wait_for_grid_in_front();    // (what is above depends on the operands alone)
    if (kGrads && run + 1 < runs) {
#pragma unroll
        for (int nj = 0; nj < 8; ++nj) {
            const float2 a = *reinterpret_cast<const float2*>(run_slot(dr, dk, base, stride, run, row_u, 8 * nj + 2 * q));
            const float2 b = *reinterpret_cast<const float2*>(run_slot(dr, dk, base, stride, run, row_d, 8 * nj + 2 * q));
            acc[nj][0] = a.x; acc[nj][1] = a.y; acc[nj][2] = b.x; acc[nj][3] = b.y;
        }
    } else {
#pragma unroll
        for (int nj = 0; nj < 8; ++nj)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[nj][e] = 0.f;
    }
    auto load_cotangent = [&](float (*m)[4]) {
#pragma unroll
        for (int nj = 0; nj < 8; ++nj) {
            const bf* p = ds_out + (size_t)bh * kN * kN + 8 * nj + 2 * q;
            const uint32_t a = *reinterpret_cast<const uint32_t*>(p + row_u * kN), b = *reinterpret_cast<const uint32_t*>(p + row_d * kN);
            m[nj][0] = __uint_as_float(low(a)); m[nj][1] = __uint_as_float(high(a));
            m[nj][2] = __uint_as_float(low(b)); m[nj][3] = __uint_as_float(high(b));
        }
    };
    const int cp = lane * 2, qt = warp;
    float2 uu = make_float2(0.f, 0.f);
    if (kGrads) uu = make_float2(__bfloat162float(u[(size_t)h * kN + cp]), __bfloat162float(u[(size_t)h * kN + cp + 1]));
    const float u_row[2] = {__bfloat162float(u[(size_t)h * kN + row_u]), __bfloat162float(u[(size_t)h * kN + row_d])};
    float dw_acc[2] = {0.f, 0.f}, du_acc[2] = {0.f, 0.f};       // of rows row_u, row_d: d * dd, and du
    __syncthreads();

    for (int c = kRunChunks - 1; c >= 0; --c) {
        const int t0 = t_run + c * kC, n = min(kC, Tlen - t0);
        const bf(*rr)[kPitch] = sm.r;
        const bf(*kk)[kPitch] = sm.k;
        const bf* const vv = &sm.v[0][0];
        const bf* const gy = &sm.dy[0][0];
        r_next.put(sm.r);
        dy_next.put(sm.dy);
        if (kGrads) { k_next.put(sm.k); v_next.put(sm.v); }
        __syncthreads();
        if (c > 0) fetch(t0 - kC);
        if (n <= 0) {
            __syncthreads();
            continue;
        }
        const uint32_t starts = sm.starts[c];
        const bool inside = ds_out != nullptr && L > t0 && L <= t0 + n;    // the returned state's cotangent enters behind token L - 1
        if (inside && L == t0 + n) {
            float m[8][4];
            load_cotangent(m);
#pragma unroll
            for (int nj = 0; nj < 8; ++nj)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[nj][e] += m[nj][e];
        }
        if (kGrads && starts != 0) {
            const int at = (tid >> 3) * kPitch + (tid & 7) * 8;
            if (odd_tiles(acc) || odd_rows(&sm.r[0][0] + at) || odd_rows(&sm.k[0][0] + at) || odd_rows(vv + at) || odd_rows(gy + at)) odd_heads[bh] = 1;
        }
        // ---- operand tiles
        auto hats = [&](int hi) {                  // K^ of a state gradient that stands behind token hi - 1
#pragma unroll
            for (int tt = 0; tt < 4; ++tt) {
                const int t = 4 * qt + tt;
                const bool last = t < hi && (starts & bits(t + 1, hi)) == 0;
                const uint32_t k2 = *reinterpret_cast<const uint32_t*>(&kk[t][cp]);
                const float2 ph = *reinterpret_cast<const float2*>(&sm.pw.p[last ? hi - 1 - t : 0][cp]);
                *reinterpret_cast<float2*>(&sm.kh[t][cp]) =
                    last ? make_float2(__uint_as_float(low(k2)) * ph.x, __uint_as_float(high(k2)) * ph.y) : make_float2(0.f, 0.f);
            }
        };
        float s1[4], s2[4];
#pragma unroll
        for (int tt = 0; tt < 4; ++tt) {
            const int t = 4 * qt + tt;
            const bool first = t < n && (starts & bits(0, t + 1)) == 0;
            const uint32_t r2 = *reinterpret_cast<const uint32_t*>(&rr[t][cp]);
            const float2 rf = make_float2(__uint_as_float(low(r2)), __uint_as_float(high(r2)));
            const float2 p0 = *reinterpret_cast<const float2*>(&sm.pw.p[first ? t : 0][cp]);
            *reinterpret_cast<float2*>(&sm.r0[t][cp]) = first ? make_float2(rf.x * p0.x, rf.y * p0.y) : make_float2(0.f, 0.f);
            if (kGrads) {
                const uint32_t k2 = *reinterpret_cast<const uint32_t*>(&kk[t][cp]);
                const float2 kf = make_float2(__uint_as_float(low(k2)), __uint_as_float(high(k2)));
                const int em = t - 1 - kMid;
                *reinterpret_cast<float2*>(&sm.rt[t][cp]) = t == 0 ? make_float2(0.f, 0.f) : make_float2(rf.x * sm.pw.at(em, cp), rf.y * sm.pw.at(em, cp + 1));
                *reinterpret_cast<float2*>(&sm.kt[t][cp]) = make_float2(kf.x * sm.pw.at(kMid - t, cp), kf.y * sm.pw.at(kMid - t, cp + 1));
                const uint32_t v2 = *reinterpret_cast<const uint32_t*>(vv + t * kPitch + cp), g2 = *reinterpret_cast<const uint32_t*>(gy + t * kPitch + cp);
                s1[tt] = __uint_as_float(low(v2)) * __uint_as_float(low(g2)) + __uint_as_float(high(v2)) * __uint_as_float(high(g2));
                s2[tt] = rf.x * uu.x * kf.x + rf.y * uu.y * kf.y;
            }
        }
        if (kGrads) {
#pragma unroll
            for (int tt = 0; tt < 4; ++tt) {
#pragma unroll
                for (int m = 1; m < 32; m <<= 1) {
                    s1[tt] += __shfl_xor_sync(0xffffffffu, s1[tt], m);
                    s2[tt] += __shfl_xor_sync(0xffffffffu, s2[tt], m);
                }
                if (lane == 0) { sm.dyv[4 * qt + tt] = s1[tt]; sm.ruk[4 * qt + tt] = s2[tt]; }
            }
            hats(n);
        }
        float dv_acc[2][4], dk_acc[2][4];          // dv: rows s, columns j = 16 warp + ...; dk^T: rows i, columns s
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) dv_acc[nt][e] = dk_acc[nt][e] = 0.f;
        const float* const S = ckpt + ((size_t)bh * nC + run * kRunChunks + c) * kN * kN;
        // what a state gradient m behind token hi - 1 gives dk, dv and dw, and (returned in m) the one in front of the chunk
        auto apply = [&](float (*m)[4], int hi) {
            const bool keep = (starts & bits(0, hi)) == 0;
            if (kGrads) {
#pragma unroll
                for (int nj = 0; nj < 8; ++nj) {
                    *reinterpret_cast<float2*>(&sm.ds[row_u][8 * nj + 2 * q]) = make_float2(m[nj][0], m[nj][1]);
                    *reinterpret_cast<float2*>(&sm.ds[row_d][8 * nj + 2 * q]) = make_float2(m[nj][2], m[nj][3]);
                }
                __syncthreads();
                if (m == acc) {                    // the operand tiles are complete: this warp's quarter of the 16 x 16 products
                    float da[2][4], dat[2][4], at[2][4];
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                        for (int e = 0; e < 4; ++e) da[nt][e] = dat[nt][e] = at[nt][e] = 0.f;
#pragma unroll
                    for (int kq = 0; kq < 2; ++kq) {
                        const int ks = 2 * warp + kq;
                        const A2 ka = rows_left(&sm.kt[0][0], kPitch, ks, g, q);
                        const A1 va = raw_rows_left(vv, ks, g, q), ga = raw_rows_left(gy, ks, g, q);
#pragma unroll
                        for (int nt = 0; nt < 2; ++nt) {
                            mma(dat[nt], va, raw_rows_right(gy, nt, ks, g, q));
                            mma(da[nt], ga, raw_rows_right(vv, nt, ks, g, q));
                            mma(at[nt], ka, rows_right(&sm.rt[0][0], kPitch, nt, ks, g, q));
                        }
                    }
                    sm.sums[0].put(warp, lane, da);
                    sm.sums[1].put(warp, lane, dat);
                    sm.sums[2].put(warp, lane, at);
                }
                float p2[2][4];
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int e = 0; e < 4; ++e) p2[nt][e] = 0.f;
#pragma unroll
                for (int ks = 0; ks < 8; ++ks) {
                    const A2 ma = as_left(m[ks]), ka = rows_left(&sm.kh[0][0], kPitch, ks, g, q);
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) {
                        mma(p2[nt], ma, raw_rows_right(vv, nt, ks, g, q));
                        mma(dv_acc[nt], ka, cols_right(&sm.ds[0][0], kPitchT, ks, 16 * warp + 8 * nt, g, q));
                    }
                }
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int s = 8 * nt + 2 * q + (e & 1), i = e < 2 ? row_u : row_d;
                        const bool last = s < hi && (starts & bits(s + 1, hi)) == 0;
                        const float x = last ? p2[nt][e] * sm.pw.p[hi - 1 - s][i] : 0.f;
                        dk_acc[nt][e] += x;
                        if (last) dw_acc[e >> 1] = fmaf((float)(hi - 1 - s) * x, __bfloat162float(kk[s][i]), dw_acc[e >> 1]);
                    }
                if (keep) {
                    float du = 0.f, dd = 0.f;
#pragma unroll
                    for (int nj = 0; nj < 8; ++nj) {
                        const float2 a = *reinterpret_cast<const float2*>(S + row_u * kN + 8 * nj + 2 * q), b = *reinterpret_cast<const float2*>(S + row_d * kN + 8 * nj + 2 * q);
                        du = fmaf(m[nj][0], a.x, fmaf(m[nj][1], a.y, du));
                        dd = fmaf(m[nj][2], b.x, fmaf(m[nj][3], b.y, dd));
                    }
                    dw_acc[0] = fmaf((float)hi * sm.pw.p[hi][row_u], du, dw_acc[0]);
                    dw_acc[1] = fmaf((float)hi * sm.pw.p[hi][row_d], dd, dw_acc[1]);
                }
            }
            const float fu = sm.pw.p[hi][row_u], fd = sm.pw.p[hi][row_d];
#pragma unroll
            for (int nj = 0; nj < 8; ++nj)
#pragma unroll
                for (int e = 0; e < 4; ++e) m[nj][e] = keep ? m[nj][e] * (e < 2 ? fu : fd) : 0.f;
        };
        if (!kGrads) __syncthreads();
        apply(acc, n);
        if (inside && L < t0 + n) {
            float m[8][4];
            load_cotangent(m);
            if (kGrads) {
                __syncthreads();                   // the first one's tiles have been read
                hats(L - t0);
            }
            apply(m, L - t0);
#pragma unroll
            for (int nj = 0; nj < 8; ++nj)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[nj][e] += m[nj][e];
        }
        // ---- dS in front of the chunk: + R0^T dY
#pragma unroll
        for (int kt = 0; kt < 2; ++kt) {
            const A2 ra = cols_left(&sm.r0[0][0], kPitchT, kt, i0, g, q);
#pragma unroll
            for (int nj = 0; nj < 8; ++nj) mma(acc[nj], ra, raw_cols_right(gy, kt, 8 * nj, g, q));
        }
        if (kGrads) {
            __syncthreads();                       // the quarters are complete
            float p1[2][4], da[2][4], dat[2][4], at[2][4];     // (S dY^T): rows i, columns t; dA: t, s; dA^T: s, t; A^T: s, t
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) p1[nt][e] = 0.f;
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
                const A2 sa = rows_left(S + (size_t)i0 * kN, kN, ks, g, q);
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) mma(p1[nt], sa, raw_rows_right(gy, nt, ks, g, q));
            }
            sm.sums[0].sum(lane, da);
            sm.sums[1].sum(lane, dat);
            sm.sums[2].sum(lane, at);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int row = g + 8 * (e >> 1), col = 8 * nt + 2 * q + (e & 1);
                    auto pair = [&](int t, int s) { return s < t && t < n && (starts & bits(s + 1, t + 1)) == 0; };
                    da[nt][e] = pair(row, col) ? da[nt][e] : 0.f;
                    dat[nt][e] = pair(col, row) ? dat[nt][e] : 0.f;
                    at[nt][e] = pair(col, row) ? at[nt][e] : row == col && row < n ? sm.ruk[row] : 0.f;
                }
            float drt[2][4], dkt[2][4];            // dR~^T: rows i, columns t; dK~^T: rows i, columns s
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) drt[nt][e] = dkt[nt][e] = 0.f;
#pragma unroll
            for (int kt = 0; kt < 2; ++kt) {
                const A2 aa = as_left(at[kt]), ka = cols_left(&sm.kt[0][0], kPitch, kt, i0, g, q), ra = cols_left(&sm.rt[0][0], kPitch, kt, i0, g, q);
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    mma(dv_acc[nt], aa, raw_cols_right(gy, kt, 16 * warp + 8 * nt, g, q));
                    mma(drt[nt], ka, as_right(da[kt], nt));
                    mma(dkt[nt], ra, as_right(dat[kt], nt));
                }
            }
            __syncthreads();                       // ... and read: their room takes the results
            // ---- dr, dk, and their shares of dw and du
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int t = 8 * nt + 2 * q + (e & 1), up = e >> 1, i = up ? row_d : row_u;
                    if (t < n) {
                        const bool first = (starts & bits(0, t + 1)) == 0;
                        const float rv = __bfloat162float(rr[t][i]), kv = __bfloat162float(kk[t][i]), dyv = sm.dyv[t];
                        const float x0 = first ? p1[nt][e] * sm.pw.p[t][i] : 0.f, x1 = t > 0 ? drt[nt][e] * sm.pw.at(t - 1 - kMid, i) : 0.f;
                        const float z = dkt[nt][e] * sm.pw.at(kMid - t, i);
                        dw_acc[up] += rv * ((float)t * x0 + (float)(t - 1) * x1) - (float)t * kv * z;
                        du_acc[up] = fmaf(rv * kv, dyv, du_acc[up]);
                        sm.out[0][t][i] = __float2bfloat16_rn(x0 + x1 + u_row[up] * kv * dyv);
                        sm.out[1][t][i] = __float2bfloat16_rn(dk_acc[nt][e] + z + u_row[up] * rv * dyv);
                    }
                    const int s = g + 8 * up, j = 16 * warp + 8 * nt + 2 * q + (e & 1);
                    sm.out[2][s][j] = __float2bfloat16_rn(dv_acc[nt][e]);
                }
            __syncthreads();
            const int row = tid >> 3, piece = (tid & 7) * 8;
            if (row < n) {
                const size_t to = base + (size_t)(t0 + row) * stride + piece;
                *reinterpret_cast<uint4*>(dr + to) = *reinterpret_cast<const uint4*>(&sm.out[0][row][piece]);
                *reinterpret_cast<uint4*>(dk + to) = *reinterpret_cast<const uint4*>(&sm.out[1][row][piece]);
                *reinterpret_cast<uint4*>(dv + to) = *reinterpret_cast<const uint4*>(&sm.out[2][row][piece]);
            }
        }
        __syncthreads();                           // the chunk's tiles have been read
    }
    if (!kGrads) {
#pragma unroll
        for (int nj = 0; nj < 8; ++nj) {
            *reinterpret_cast<float2*>(run_slot(dr, dk, base, stride, run - 1, row_u, 8 * nj + 2 * q)) = make_float2(acc[nj][0], acc[nj][1]);
            *reinterpret_cast<float2*>(run_slot(dr, dk, base, stride, run - 1, row_d, 8 * nj + 2 * q)) = make_float2(acc[nj][2], acc[nj][3]);
        }
        return;
    }
#pragma unroll
    for (int up = 0; up < 2; ++up) {               // over the four lanes of a row
        const int i = up ? row_d : row_u;
        float a = dw_acc[up], b = du_acc[up];
        a += __shfl_xor_sync(0xffffffffu, a, 1); a += __shfl_xor_sync(0xffffffffu, a, 2);
        b += __shfl_xor_sync(0xffffffffu, b, 1); b += __shfl_xor_sync(0xffffffffu, b, 2);
        if (q == 0) {
            part[(size_t)blockIdx.x * 2 * kN + i] = a / sm.pw.p[1][i];
            part[(size_t)blockIdx.x * 2 * kN + kN + i] = b;
        }
    }
    if (run == 0) {
        if (L == 0 && ds_out != nullptr) {
            float m[8][4];
            load_cotangent(m);
#pragma unroll
            for (int nj = 0; nj < 8; ++nj)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[nj][e] += m[nj][e];
        }
#pragma unroll
        for (int nj = 0; nj < 8; ++nj) {
            bf* p = ds0 + (size_t)bh * kN * kN + 8 * nj + 2 * q;
            *reinterpret_cast<__nv_bfloat162*>(p + row_u * kN) = __floats2bfloat162_rn(acc[nj][0], acc[nj][1]);
            *reinterpret_cast<__nv_bfloat162*>(p + row_d * kN) = __floats2bfloat162_rn(acc[nj][2], acc[nj][3]);
        }
    }
}

// The runs' shares of dw and du of one head, added in order.
__global__ void __launch_bounds__(128)
wkv5_sum_runs_kernel(int H, int runs, const bf* __restrict__ w, const float* part, float* __restrict__ dw, float* __restrict__ du) {
    const int bh = blockIdx.x, i = threadIdx.x & 63;
    let_next_in();
    wait_for_grid_in_front();
    if (!in_domain(w + (size_t)(bh % H) * kN)) return;
    float s = 0.f;
    for (int rn = 0; rn < runs; ++rn) s += part[((size_t)bh * runs + rn) * 2 * kN + threadIdx.x];
    (threadIdx.x < kN ? dw : du)[(size_t)bh * kN + i] = s;
}

int runs_of(int T) { return (T + kRun - 1) / kRun; }
}  // namespace

// Behind a residual's checkpoints: the runs' shares of dw and du, and a word per head.
size_t wkv5_exact_partial_bytes(int B, int T, int H) { return (size_t)B * H * (runs_of(T) * (size_t)(2 * kN) * sizeof(float) + sizeof(int)); }
// The words per head (see odd() above) of a call with this residual, or with this workspace.
int* wkv5_odd_heads(int B, int T, int H, void* residual, void* workspace) {
    const size_t BH = (size_t)B * H;
    char* const base = static_cast<char*>(residual != nullptr ? residual : workspace);
    const size_t behind = residual != nullptr ? ((size_t)((T + kC - 1) / kC) * kN * kN + (size_t)runs_of(T) * 2 * kN) : (size_t)runs_of(T) * kN * kN;
    return reinterpret_cast<int*>(base + BH * behind * sizeof(float));
}

// Rows travel in 16-byte pieces here (8 bytes in the token-sequential kernels), and the scan keeps a byte per run in shared memory.
bool wkv5_exact_takes(int T, std::initializer_list<const void*> operands) {
    uintptr_t bits = 0;
    for (const void* p : operands) bits |= reinterpret_cast<uintptr_t>(p);
    return (bits & 15u) == 0 && runs_of(T) <= 48 * 1024;
}

// What a call without a residual needs to keep: the states between its runs, and a word per head.
size_t wkv5_states_bytes(int B, int T, int H) { return (size_t)B * H * (runs_of(T) * (size_t)kN * kN * sizeof(float) + sizeof(int)); }

// Exactly one of `residual` (the checkpoints, a state per chunk, stay there for the backward) and `workspace` is given.
int wkv5_exact_fwd(cudaStream_t st, int B, int T, int H, const void* r, const void* k, const void* v, const void* w, const void* u,
                   const void* s0, const uint32_t* length, const uint8_t* ns, void* y, void* s_out, void* residual, int* residual_mark,
                   void* workspace) {
    static DeviceOnce attr;
    if (!attr.ok([]() {
            cudaError_t e = cudaFuncSetAttribute(wkv5_fwd_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FwdSmem5));
            if (e == cudaSuccess) e = cudaFuncSetAttribute(wkv5_fwd_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FwdSmem5));
            return e;
        }))
        return B200WKV_ELAUNCH;
    const int runs = runs_of(T), heads = B * H, per_run = residual != nullptr ? kRunChunks : 1;
    const int n_states = residual != nullptr ? (T + kC - 1) / kC : runs;
    float* const states = (float*)(residual != nullptr ? residual : workspace);
    int* const odd_heads = wkv5_odd_heads(B, T, H, residual, workspace);
    cudaError_t e = cudaSuccess;
    auto launch = [&](bool first, auto kern, int n) {
        e = launch_in_chain(first, kern, heads * n, 128, sizeof(FwdSmem5), st, T, H, n, n_states, per_run, (const bf*)r, (const bf*)k, (const bf*)v, (const bf*)w,
                            (const bf*)u, (const bf*)s0, length, ns, (bf*)y, (bf*)s_out, states, odd_heads, residual_mark);
    };
    if (runs > 1) launch(true, wkv5_fwd_kernel<false>, runs - 1);
    if (e == cudaSuccess)
        e = launch_in_chain(runs == 1, wkv5_scan_kernel<true>, dim3(heads, kN * kN / 1024), 256, runs, st, T, H, runs, n_states, per_run, (const bf*)w,
                            (const bf*)s0, ns, states, odd_heads, (bf*)nullptr, (bf*)nullptr);
    if (e == cudaSuccess) launch(false, wkv5_fwd_kernel<true>, runs);
    return e == cudaSuccess ? B200WKV_OK : B200WKV_ELAUNCH;
}

int wkv5_exact_bwd(cudaStream_t st, int B, int T, int H, const void* r, const void* k, const void* v, const void* w, const void* u,
                   const uint32_t* length, const uint8_t* ns, const void* dy, const void* ds_out, void* residual, void* partial,
                   void* dr, void* dk, void* dv, void* dw, void* du, void* ds0) {
    static DeviceOnce attr;
    if (!attr.ok([]() {
            cudaError_t e = cudaFuncSetAttribute(wkv5_bwd_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BwdSmem5));
            if (e == cudaSuccess) e = cudaFuncSetAttribute(wkv5_bwd_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BwdSmem5));
            return e;
        }))
        return B200WKV_ELAUNCH;
    const int runs = runs_of(T), heads = B * H;
    int* const odd_heads = wkv5_odd_heads(B, T, H, residual, nullptr);
    cudaError_t e = cudaSuccess;
    auto launch = [&](bool first, auto kern, int n) {
        e = launch_in_chain(first, kern, heads * n, 128, sizeof(BwdSmem5), st, T, H, runs, (const bf*)r, (const bf*)k, (const bf*)v, (const bf*)w, (const bf*)u,
                            length, ns, (const bf*)dy, (const bf*)ds_out, (const float*)residual, odd_heads, (bf*)dr, (bf*)dk, (bf*)dv, (float*)partial,
                            (bf*)ds0);
    };
    if (runs > 1) {
        launch(true, wkv5_bwd_kernel<false>, runs - 1);
        if (e == cudaSuccess)
            e = launch_behind(wkv5_scan_kernel<false>, dim3(heads, kN * kN / 1024), 256, runs, st, T, H, runs, 0, 0, (const bf*)w, (const bf*)nullptr, ns,
                              (float*)nullptr, (int*)nullptr, (bf*)dr, (bf*)dk);
    }
    if (e == cudaSuccess) launch(runs == 1, wkv5_bwd_kernel<true>, runs);
    if (e == cudaSuccess) e = launch_behind(wkv5_sum_runs_kernel, heads, 128, 0, st, H, runs, (const bf*)w, (const float*)partial, (float*)dw, (float*)du);
    return e == cudaSuccess ? B200WKV_OK : B200WKV_ELAUNCH;
}

}  // namespace b200wkv
