// RWKV-7 in fp32 arithmetic, 16 tokens at a time: everything that does not depend on the state for all chunks side by side,
// and a chain over the chunks whose step is two products of 16 tokens with the state instead of 16 dependent tokens.
//
// Per chunk, with P_t the decay of the tokens in front of t and [s, t] that of the tokens s..t (products; nothing is divided by
// a decay, so none is too strong), all per key channel:
//   beta_ts = sum_j b_s a_t (s, t)      kappa_ts = sum_j k_s a_t (s, t)       s < t     (exclusive ranges)
//   rho_ts  = sum_j b_s r_t (s, t]      sigma_ts = sum_j k_s r_t (s, t]       s <= t
//   a~_t = a_t P_t    r~_t = r_t P_t+1    b^_s = b_s (s, C)    k^_s = k_s (s, C)
// Forward (S0 = the entering state, s_t = S_{t-1} a_t, z_t its part that comes from S0):
//   W~ = (I - beta)^-1 a~        z = W~ S0^T        u = (I - beta)^-1 kappa V           s = z + u
//   S_C = S0 diag(P_C) + z^T b^ + D      D = u^T b^ + V^T k^
//   y = R- S0^T + y'                     R- = r~ + rho W~     y' = rho u + sigma V
// Backward (G = the gradient of the state behind the chunk, g_t = the gradient of s_t):
//   B~ = (I - beta^T)^-1 b^      z = B~ G^T         u = (I - beta^T)^-1 rho^T dY         g = z + u
//   G' = G diag(P_C) + z^T a~ + D'       D' = u^T a~ + dY^T r~
// and with s and g of every token known, the gradients of a chunk need no sum over the state's rows or columns before the next
// token: wkv7_fp32_grads_kernel walks S forward and dS back elementwise.
//
// The token-by-token chain (wkv7_chain.cu) takes 0.12-0.15 us per token whatever else the device does, the chain here 0.6-1.1 us per
// 16 tokens, and what is taken out of it fills the device.  Forward of 8 heads, T=256: 32.8 -> 22.5 us (6 before the chain, 13
// in it, 3 behind); forward and backward of 24 heads, T=512: 280 -> 155 us, where the gradients
// were 131 us of sums over rows and columns that every token waited for.  Errors against 64 bits (without flags / a flag every 128
// tokens), token by token and here: outputs 1.02e-7 / 1.02e-7 and 0.98e-7 / 0.98e-7, state 0.77e-7 / 0.76e-7 and 0.79e-7 / 0.76e-7, the
// nearest and the farthest gradient 0.96-1.39e-7 / 0.95-1.39e-7 and 0.96-1.41e-7 / 0.96-1.40e-7.
//
// Chunks with a start flag behind their first token, those that `length` cuts and those of fewer than
// 16 tokens are walked token by token inside the chain kernel (its sums in another order than wkv7_chain.cu's): a flag drops the state whatever it
// holds.  Semantics: BaseRWKV.inner_loop of jaxrwkv (src/jaxrwkv/rwkv7.py:199-220) and its reverse.
#include "common.cuh"
#include "device_once.cuh"
#include "tc05.cuh"
#include "wkv7_exact.cuh"

namespace b200wkv {

int* wkv7_chunk_status_word();

namespace {

constexpr int kC = kExactChunk;
constexpr int kTile = kC * kN;                       // floats of a tile [token][channel]

// What the chain reads of a chunk lies at left / right / decay + head * head_stride + chunk * chunk_stride: forward W~, b^, P_C,
// backward B~, a~, P_C.
struct Tiles {
    float *left, *right, *rbar, *decay;              // rbar: forward only
    size_t head_stride, chunk_stride;
};
struct Operands {
    int T, H;
    const float *w, *r, *k, *v, *a, *b;              // backward: v is dy, which may be NULL (zero)
    const uint32_t* length;
    const uint8_t* new_starts;
};

// How a chunk is done: whole, whole from a zero state (a flag on its first token), or token by token.
enum { kWhole = 0, kFresh = 1, kWalked = 2 };
__device__ __forceinline__ int kind_of(uint32_t starts, int t0, int T, int L) {
    if (t0 + kC > T || (starts & ~1u) != 0 || (L > t0 && L < t0 + kC)) return kWalked;
    return (int)(starts & 1u);
}

__device__ __forceinline__ float4 at4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void put4(float* p, const float4& x) { *reinterpret_cast<float4*>(p) = x; }
// v[i] summed over 16 lanes, the sum of v[lane % 16] returned.  What the last three additions round off is added at the end: the pair
// sums go into all rows of the state, and without this s would be 4 % less accurate than in the token-by-token recurrence.
__device__ __forceinline__ float rounded_off(float x, float y, float sum) {     // exact: x + y = sum + this
    const float z = sum - x;
    return (x - (sum - z)) + (y - z);
}
__device__ __forceinline__ float transpose_sum16(float* v, int lane) {
    float low[4];
#pragma unroll
    for (int m = 8; m > 0; m >>= 1) {
        const bool up = lane & m;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (i < m) {
                const float keep = up ? v[i + m] : v[i], got = __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + m], m);
                v[i] = keep + got;
                const float off = rounded_off(keep, got, v[i]);
                if (m == 4) low[i] = off;
                if (m < 4) low[i] = (up ? low[i + m] : low[i]) + __shfl_xor_sync(0xffffffffu, up ? low[i] : low[i + m], m) + off;
            }
    }
    return fabsf(v[0]) < __int_as_float(0x7f800000) ? v[0] + low[0] : v[0];
}
struct Row4 { Pair lo, hi; };                        // four columns
__device__ __forceinline__ Row4 row4(const float* p) {
    const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(p);
    return Row4{Pair{u.x}, Pair{u.y}};
}
__device__ __forceinline__ void put_row4(float* p, const Row4& x) { *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(x.lo.u, x.hi.u); }
__device__ __forceinline__ float dot(const Row4& x, const Row4& y) {
    const float2 s = unpack(fma2(x.hi, y.hi, mul2(x.lo, y.lo)));
    return s.x + s.y;
}
__device__ __forceinline__ Row4 mul(const Row4& x, const Row4& y) { return Row4{mul2(x.lo, y.lo), mul2(x.hi, y.hi)}; }

// ------------------------------------------------------------------ what no state enters --------
constexpr int kPrepThreads = 256;
constexpr int kMat = kC + 4;                         // pitch of a [16][16] matrix in shared memory
struct PrepSmem {
    float w[kC][kN], a[kC][kN], b[kC][kN], k[kC][kN], r[kC][kN], v[kC][kN];
    float a4[kC][kN], r4[kC][kN];                    // a and r with the decays from the start of their block of four tokens on
    float decay4[4][kN];                             // of a whole block of four tokens
    float left[kC][kN], right[kC][kN], right2[kC][kN], rbar[kC][kN], u[kC][kN];
    // pair sums, a row per token that is summed over (solved for: beta), its columns the tokens that receive: forward [s][t],
    // backward [t][s]
    float beta[kC][kMat], kappa[kC][kMat], rho[kC][kMat], sigma[kC][kMat];
};

// acc[i] = token t0 + i, four columns: += sum over the tokens s <= t0 + i of m[s][t] x[s], from the farthest to the nearest: the
// terms grow, so that the sum rounds where it is small
__device__ __forceinline__ void times_tile(Row4 (&acc)[4], const float (*m)[kMat], const float (*x)[kN], int t0, int col) {
    auto add = [&](int s, int first) {
        const float4 f = at4(&m[s][t0]);
        const float fe[4] = {f.x, f.y, f.z, f.w};
        const Row4 g = row4(&x[s][col]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i >= first) {
                const Pair ff = pair(fe[i], fe[i]);
                acc[i].lo = fma2(ff, g.lo, acc[i].lo);
                acc[i].hi = fma2(ff, g.hi, acc[i].hi);
            }
    };
#pragma unroll 4
    for (int s = 0; s < t0; ++s) add(s, 0);
#pragma unroll
    for (int e = 0; e < 4; ++e) add(t0 + e, e);
}

// One CTA per chunk.  `slots` receives D, `sums` (NULL: not wanted) u, y the outputs from a zero state.  Bound by
// shared-memory reads and, for the pair sums, by issue, so that threads have tiles of the products and two tokens of the pair sums:
// 3.2 us per chunk and SM forward, 2.6 backward (one token and 4 x 4 of D per thread: 4.8).
template <bool kForward>
__global__ void __launch_bounds__(kPrepThreads, 3)
wkv7_fp32_prepare_kernel(const Operands op, const Tiles tiles, float* __restrict__ slots, float* __restrict__ sums, float* __restrict__ y) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    PrepSmem& sm = *reinterpret_cast<PrepSmem*>(smem_raw);
    const int nC = (op.T + kC - 1) / kC, bh = blockIdx.x / nC, c = blockIdx.x % nC, bi = bh / op.H, h = bh % op.H;
    const int tid = threadIdx.x, t0 = c * kC, row = tid >> 4, lane16 = tid & 15, col = lane16 * 4;
    const int L = min((int)op.length[bi], op.T);
    const bool flag = tid > 0 && tid < kC && t0 + tid < op.T && op.new_starts[(size_t)bi * op.T + t0 + tid] != 0;
    const size_t seq = (size_t)bi * op.T * op.H * kN + (size_t)h * kN, tok = (size_t)op.H * kN;
    const size_t mine = seq + (size_t)(t0 + row) * tok + col;
    if (__syncthreads_or(flag) || kind_of(0, t0, op.T, L) == kWalked) {      // only the decays, which every warp of the chain needs
        if (t0 + row < op.T) put4(tiles.left + bh * tiles.head_stride + c * tiles.chunk_stride + row * kN + col, decay4(at4(op.w + mine)));
        return;
    }
    {
        const float4 w = at4(op.w + mine), a = at4(op.a + mine), b = at4(op.b + mine), r = at4(op.r + mine);
        const float4 k = kForward ? at4(op.k + mine) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 v = op.v != nullptr ? at4(op.v + mine) : make_float4(0.f, 0.f, 0.f, 0.f);
        put4(&sm.w[row][col], decay4(w));
        put4(&sm.a[row][col], a);
        put4(&sm.b[row][col], b);
        put4(&sm.r[row][col], r);
        if (kForward) put4(&sm.k[row][col], k);
        put4(&sm.v[row][col], v);
    }
    __syncthreads();
    // The decay over a stretch of tokens is a product inside a block of four, whole blocks, and a product inside another block:
    // half the roundings of one product after the other, and the pair sums need no factor per token and pair.
    {
        const int q = tid >> 6, j = tid & 63;
        float p = 1.f, z = 1.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int t = 4 * q + e;
            sm.a4[t][j] = sm.a[t][j] * p;
            p *= sm.w[t][j];
            sm.r4[t][j] = sm.r[t][j] * p;
        }
        sm.decay4[q][j] = p;
#pragma unroll
        for (int e = 3; e >= 0; --e) {
            const int t = 4 * q + e;
            (kForward ? sm.right : sm.left)[t][j] = sm.b[t][j] * z;      // (up to the end of the block)
            if (kForward) sm.right2[t][j] = sm.k[t][j] * z;
            z *= sm.w[t][j];
        }
    }
    __syncthreads();
    const size_t tile_at = bh * tiles.head_stride + c * tiles.chunk_stride;
    if (tid < 128) {
        // The pair sums: 16 lanes with four channels each carry b (and k) of tokens s and s + 8 on through the decays of the
        // tokens behind.  Four tokens' sums at a time are added up over the lanes, 16 values for 16 lanes.
        constexpr int kKinds = kForward ? 2 : 1;     // b, k
        const int block = row >> 2;                  // of token s (of s + 8: + 2); the same for a whole warp
        Row4 g[2][kKinds];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            g[i][0] = row4(&sm.b[row + 8 * i][col]);
            if (kForward) g[i][kKinds - 1] = row4(&sm.k[row + 8 * i][col]);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            float x[2][8 * kKinds];                  // [kind][a, r][token]
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                if (q < 2 * i) continue;             // in front of all tokens s + 8
                const int s = row + 8 * i;
                if (q == block + 2 * i) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int t = 4 * q + e;
                        const Row4 at = row4(&sm.a[t][col]), wt = row4(&sm.w[t][col]), rt = row4(&sm.r[t][col]);
#pragma unroll
                        for (int m = 0; m < kKinds; ++m) {
                            x[i][8 * m + e] = t > s ? dot(g[i][m], at) : 0.f;
                            if (t > s) g[i][m] = mul(g[i][m], wt);
                            x[i][8 * m + 4 + e] = t >= s ? dot(g[i][m], rt) : 0.f;
                        }
                    }
                } else if (q > block + 2 * i) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const Row4 at = row4(&sm.a4[4 * q + e][col]), rt = row4(&sm.r4[4 * q + e][col]);
#pragma unroll
                        for (int m = 0; m < kKinds; ++m) {
                            x[i][8 * m + e] = dot(g[i][m], at);
                            x[i][8 * m + 4 + e] = dot(g[i][m], rt);
                        }
                    }
                    const Row4 wt = row4(&sm.decay4[q][col]);
#pragma unroll
                    for (int m = 0; m < kKinds; ++m) g[i][m] = mul(g[i][m], wt);
                } else {
#pragma unroll
                    for (int e = 0; e < 8 * kKinds; ++e) x[i][e] = 0.f;
                }
            }
            auto keep = [&](int s, int kind, int of_r, int t, float f) {
                float (*const to)[kMat] = kind == 0 ? (of_r ? sm.rho : sm.beta) : (of_r ? sm.sigma : sm.kappa);
                if (kForward) to[s][t] = f; else to[t][s] = f;
            };
            if (kForward) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float f = q < 2 * i ? 0.f : transpose_sum16(x[i], lane16);
                    keep(row + 8 * i, lane16 >> 3, (lane16 >> 2) & 1, 4 * q + (lane16 & 3), f);
                }
            } else {
                float z[16];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    z[e] = x[0][e];
                    z[8 + e] = q < 2 ? 0.f : x[1][e];
                }
                keep(row + 8 * (lane16 >> 3), 0, (lane16 >> 2) & 1, 4 * q + (lane16 & 3), transpose_sum16(z, lane16));
            }
        }
    } else if (tid < 128 + kN) {                     // right-hand sides and operands in front of the chunk's tokens
        const int j = tid - 128;
        float p = 1.f;
#pragma unroll
        for (int t = 0; t < kC; ++t) {
            if (t > 0 && t % 4 == 0) p *= sm.decay4[t / 4 - 1][j];
            (kForward ? sm.left : sm.right)[t][j] = sm.a4[t][j] * p;
            (kForward ? sm.rbar : sm.right2)[t][j] = sm.r4[t][j] * p;
        }
        tiles.decay[tile_at + j] = p * sm.decay4[3][j];
    } else {                                         // and behind them
        const int j = tid - 128 - kN;
        float p = 1.f;
#pragma unroll
        for (int t = kC - 5; t >= 0; --t) {
            if (t % 4 == 3) p *= sm.decay4[t / 4 + 1][j];
            (kForward ? sm.right : sm.left)[t][j] *= p;
            if (kForward) sm.right2[t][j] *= p;
        }
    }
    __syncthreads();
    // (I - beta) X = right-hand sides, a thread per column: W~ (B~), and u, whose right-hand side kappa V (rho^T dY) comes in on
    // the way, each token's term beside its correction
    if (tid < 2 * kN) {
        const int j = tid & (kN - 1);
        const bool of_u = tid >= kN;
        const float (*const into)[kMat] = kForward ? sm.kappa : sm.rho;
        float x[kC], own[kC];                        // (the two sums apart: each rounds at its own size)
#pragma unroll
        for (int t = 0; t < kC; ++t) own[t] = 0.f;
        if (of_u) {
#pragma unroll
            for (int t = 0; t < kC; ++t) x[t] = 0.f;
        } else {
#pragma unroll
            for (int t = 0; t < kC; ++t) x[t] = sm.left[t][j];
        }
#pragma unroll
        for (int i = 0; i < kC; ++i) {
            const int t = kForward ? i : kC - 1 - i;
            const float v = of_u ? sm.v[t][j] : 0.f;
            if (!kForward && of_u) own[t] = fmaf(into[t][t], v, own[t]);
            x[t] += own[t];
#pragma unroll
            for (int q = 0; q < kC / 4; ++q) {
                if (kForward ? 4 * q + 3 <= t : 4 * q >= t) continue;
                auto add = [&](float (&x)[kC], const float4& f, float z) {
                    const float fe[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (kForward ? 4 * q + e > t : 4 * q + e < t) x[4 * q + e] = fmaf(fe[e], z, x[4 * q + e]);
                };
                if (of_u) add(own, at4(&into[t][4 * q]), v);
                add(x, at4(&sm.beta[t][4 * q]), x[t]);
            }
        }
        float* const column = (of_u ? &sm.u[0][0] : &sm.left[0][0]) + j;
#pragma unroll
        for (int t = 0; t < kC; ++t) column[t * kN] = x[t];
    }
    __syncthreads();
    const size_t in_tile = tile_at + row * kN + col;
    put_row4(tiles.left + in_tile, row4(&sm.left[row][col]));
    put_row4(tiles.right + in_tile, row4(&sm.right[row][col]));
    if (sums != nullptr) put_row4(kForward ? sums + ((size_t)bh * op.T + t0 + row) * kN + col : sums + mine, row4(&sm.u[row][col]));
    const int quarter = (tid >> 4) & 3;              // of 64 threads: tokens 4 quarter .. + 3, columns col .. col + 3
    Row4 acc[4];
    if (kForward && tid >= 64 && tid < 128) {        // y' = sigma V + rho u
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i].lo.u = acc[i].hi.u = 0;
        Row4 of_v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) of_v[i] = acc[i];
        times_tile(acc, sm.rho, sm.u, 4 * quarter, col);
        times_tile(of_v, sm.sigma, sm.v, 4 * quarter, col);
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] = Row4{add2(acc[i].lo, of_v[i].lo), add2(acc[i].hi, of_v[i].hi)};
#pragma unroll
        for (int i = 0; i < 4; ++i) put_row4(y + seq + (size_t)(t0 + 4 * quarter + i) * tok + col, acc[i]);
    } else if (kForward && tid < 64) {               // R- = r~ + rho W~
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] = row4(&sm.rbar[4 * quarter + i][col]);
        times_tile(acc, sm.rho, sm.left, 4 * quarter, col);
#pragma unroll
        for (int i = 0; i < 4; ++i) put_row4(tiles.rbar + tile_at + (4 * quarter + i) * kN + col, acc[i]);
    } else if (tid >= 128) {                         // D, eight rows (as pairs) by four columns of it per thread
        const int i0 = ((tid - 128) >> 4) * 8;
        Pair d[4][4];
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int e = 0; e < 4; ++e) d[p][e].u = 0;
        auto add = [&](const float (*x)[kN], const float (*z)[kN], int t) {
            const Row4 x0 = row4(&x[t][i0]), x1 = row4(&x[t][i0 + 4]);
            const Pair xp[4] = {x0.lo, x0.hi, x1.lo, x1.hi};
            const float4 f = at4(&z[t][col]);
            const float fe[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const Pair ff = pair(fe[e], fe[e]);
#pragma unroll
                for (int p = 0; p < 4; ++p) d[p][e] = fma2(xp[p], ff, d[p][e]);
            }
        };
#pragma unroll 4
        for (int i = 0; i < kC; ++i) {               // from the token farthest from the end that D is at
            const int t = kForward ? i : kC - 1 - i;
            add(sm.u, sm.right, t);
            add(sm.v, sm.right2, t);
        }
        float* const to = slots + ((size_t)bh * nC + c) * (kN * kN) + i0 * kN + col;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            float2 f[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) f[e] = unpack(d[p][e]);
            put4(to + (2 * p) * kN, make_float4(f[0].x, f[1].x, f[2].x, f[3].x));
            put4(to + (2 * p + 1) * kN, make_float4(f[0].y, f[1].y, f[2].y, f[3].y));
        }
    }
}

// ------------------------------------------------------------------ the chain --------
// Rows of the state never meet, so a (sequence, head) is spread over CTAs of 2 R W rows: W computing warps of two groups of 16
// lanes, each group R rows, four columns of each row in a lane, and a warp that fetches the chunks' tiles (of a chunk that is
// walked: its raw rows) by bulk copies, five to eight chunks ahead.  A step is latency: dot products, their sums over the lanes, the way of the sums back to all
// lanes, the update, 0.65 us for one row, 0.8 for two, 1.1 for four (dealing a step's products out to more threads, with the state
// in shared memory and barriers in between, was no faster).
//
// Forward: out = the state at `length`, slots receive the state entering every chunk (0 where its first token starts anew), y the
// outputs of the chunks that are walked.  Backward: x0 the returned state's cotangent (NULL: zero), out = the gradient of the
// initial state, slots receive the gradient of the state behind every chunk (without that cotangent, where it enters there).
// Both read D from the slots first.  `sums` (forward [head][token][64], NULL: not wanted; backward like a stream) holds u and
// receives s or g.
template <int W, int R>
struct ChainSmem {
    static constexpr int kRows = 2 * R * W, kWarps = W;              // rows, computing warps of a CTA
    static constexpr int kStages = kRows <= 8 ? 8 : kRows <= 16 ? 6 : 5;      // (five of 22 KB: two CTAs per SM)
    struct Whole { float left[kC][kN], right[kC][kN], decay[kN], d[kRows][kN]; };
    struct Walked { float decay[kC][kN], a[kC][kN], b[kC][kN], r[kC][kN], k[kC][kN], v[kC][kRows]; };      // raw rows of tokens
    union Stage { Whole whole; Walked walked; } st[kStages];
    float s[kRows][kC];
    uint64_t full[kStages], empty[kStages];
    int kind[kStages];
    uint32_t starts[kStages];

    __device__ __forceinline__ void init() {
#pragma unroll
        for (int i = 0; i < kStages; ++i) {
            tc::mbar_init(&full[i], 1);
            tc::mbar_init(&empty[i], kWarps);
        }
        tc::mbar_init_fence();
    }
};

// Where a CTA is, and what of its chunks lies where
template <bool kForward>
struct Place {
    int nC, bh, part, bi, L;
    size_t seq, tok;
    __device__ __forceinline__ Place(const Operands& op, int parts)
        : nC((op.T + kC - 1) / kC), bh(blockIdx.x / parts), part(blockIdx.x % parts), bi(bh / op.H), L(min((int)op.length[bi], op.T)),
          seq((size_t)bi * op.T * op.H * kN + (size_t)(bh % op.H) * kN), tok((size_t)op.H * kN) {}
    __device__ __forceinline__ int chunk(int it) const { return kForward ? it : nC - 1 - it; }
    __device__ __forceinline__ size_t slot(int it) const { return ((size_t)bh * nC + chunk(it)) * (kN * kN); }
    // s (g) of token t, row 0
    __device__ __forceinline__ size_t sum(const Operands& op, int t) const { return kForward ? ((size_t)bh * op.T + t) * kN : seq + (size_t)t * tok; }
};

// The fetching warp (flags and lengths are the caller's: only the tiles have to be waited for).  False where a wait ran out: the
// computing warps give up as well then.
template <bool kForward, class Smem>
__device__ __forceinline__ bool fetch_chunks(Smem& sm, const Operands& op, const Tiles& tiles, const Place<kForward>& at, const float* slots) {
    const int lane = threadIdx.x & 31;
    const uint8_t* const ns = op.new_starts + (size_t)at.bi * op.T;
    constexpr int kRaw = kForward ? 4 : 3;           // streams fetched whole: a, b, r, forward k
    uint32_t ahead = 0;                              // flags of 32 chunks, one per lane
    for (int it = 0; it < at.nC; ++it) {
        const int stage = it % Smem::kStages, t0 = at.chunk(it) * kC, n = min(kC, op.T - t0);
        if ((it & 31) == 0) {
            ahead = 0;
            const int first = at.chunk(min(it + lane, at.nC - 1)) * kC;
#pragma unroll
            for (int i = 0; i < kC; ++i)
                if (first + i < op.T && ns[first + i] != 0) ahead |= 1u << i;
        }
        const uint32_t starts = __shfl_sync(0xffffffffu, ahead, it & 31);
        const int kind = kind_of(starts, t0, op.T, at.L);
        if (it == 0) wait_for_grid_in_front();
        if (it >= Smem::kStages && !tc::mbar_wait(&sm.empty[stage], (it / Smem::kStages - 1) & 1)) return false;
        uint64_t* const bar = &sm.full[stage];
        if (lane == 0) {
            sm.kind[stage] = kind;
            sm.starts[stage] = starts;
            tc::mbar_expect_tx(bar, (uint32_t)((kind == kWalked ? n * ((kRaw + 1) * kN + (op.v != nullptr ? Smem::kRows : 0))
                                                                : 2 * kTile + kN + Smem::kRows * kN) * 4));
        }
        __syncwarp();
        const size_t tile = at.bh * tiles.head_stride + at.chunk(it) * tiles.chunk_stride;
        if (kind == kWalked) {                       // a lane one token of two of the streams
            typename Smem::Walked& s = sm.st[stage].walked;
            const int t = lane & 15;
            const size_t row = at.seq + (size_t)(t0 + t) * at.tok;
            if (lane == 0) tc::bulk_load(s.decay, tiles.left + tile, (uint32_t)(n * kN * 4), bar);
            if (t < n) {
                const bool even = lane < 16;
                tc::bulk_load(even ? s.a[t] : s.b[t], (even ? op.a : op.b) + row, kN * 4, bar);
                if (even) tc::bulk_load(s.r[t], op.r + row, kN * 4, bar);
                else if (kForward) tc::bulk_load(s.k[t], op.k + row, kN * 4, bar);
                if (!even && op.v != nullptr) tc::bulk_load(s.v[t], op.v + row + at.part * Smem::kRows, Smem::kRows * 4, bar);
            }
        } else {
            typename Smem::Whole& s = sm.st[stage].whole;
            if (lane == 0) tc::bulk_load(s.left, tiles.left + tile, kTile * 4, bar);
            else if (lane == 1) tc::bulk_load(s.right, tiles.right + tile, kTile * 4, bar);
            else if (lane == 2) tc::bulk_load(s.decay, tiles.decay + tile, kN * 4, bar);
            else if (lane == 3) tc::bulk_load(s.d, slots + at.slot(it) + at.part * Smem::kRows * kN, Smem::kRows * kN * 4, bar);
        }
    }
    return true;
}

// A lane's four columns of R rows
template <int R>
struct Slice {
    Row4 x[R];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int m = 0; m < R; ++m) x[m].lo.u = x[m].hi.u = 0;
    }
    __device__ __forceinline__ void load(const float* from) {
#pragma unroll
        for (int m = 0; m < R; ++m) x[m] = row4(from + m * kN);
    }
    __device__ __forceinline__ void store(float* to) const {
#pragma unroll
        for (int m = 0; m < R; ++m) put_row4(to + m * kN, x[m]);
    }
    __device__ __forceinline__ void add(const float* from) {
#pragma unroll
        for (int m = 0; m < R; ++m) {
            const Row4 g = row4(from + m * kN);
            x[m].lo = add2(x[m].lo, g.lo);
            x[m].hi = add2(x[m].hi, g.hi);
        }
    }
};

// A chunk token by token.  What a token waits for is one sum over 16 lanes, which all rows of a lane take together; the operands of four
// tokens are in registers before the first of them, and the outputs' sums, which nothing waits for, are taken for four tokens at
// once.  Its rows come through the stages that whole chunks' tiles come through, so that they are fetched as far ahead: with one
// buffer for them apart, asked for when the walked chunk in front was done, a chunk was 5.4 us, and is 2.5 (4 heads; 81 copies to issue
// for it take as long as its tokens; four rows per lane and two CTAs per SM: 3.3 a chunk and SM).  us of a forward, before / now: 4 heads,
// T=2048, all chunks walked 701 / 332, a flag every 16 tokens 469 / 255 (the token-by-token kernel 235); 24 heads 890 / 413 and 631 / 345;
// 128 heads, T=512 319 / 214 and 283 / 210.  Fetched by 16-byte asynchronous copies: 321, but 2 % more where no chunk is walked.
template <int R>
__device__ __forceinline__ void sum16(float* x) {
#pragma unroll
    for (int bit = 1; bit < 16; bit <<= 1)
#pragma unroll
        for (int m = 0; m < R; ++m) x[m] += __shfl_xor_sync(0xffffffffu, x[m], bit);
}
template <bool kForward, int R, class Walked>
__device__ __forceinline__ void walk(Slice<R>& x, const Walked& s, const Operands& op, const Place<kForward>& at, int t0, uint32_t starts, int row, int own,
                                     int col, const float* x0, float* sums, float* y, float* out) {
    constexpr int kStep = 4;
    const int n = min(kC, op.T - t0), l = col >> 2;
    const size_t state_at = ((size_t)at.bh * kN + row) * kN + col;
    const int stop = kForward || x0 != nullptr ? at.L - 1 - t0 : -1;     // the token behind which the returned state lies
    auto axpy = [](Pair f, const Row4& a, const Row4& b) { return Row4{fma2(f, a.lo, b.lo), fma2(f, a.hi, b.hi)}; };
    auto keep_if = [](bool c, const Row4& a, const Row4& b) { return Row4{Pair{c ? a.lo.u : b.lo.u}, Pair{c ? a.hi.u : b.hi.u}}; };
    const Row4 none{Pair{0}, Pair{0}};
#pragma unroll 1
    for (int i0 = 0; i0 < n; i0 += kStep) {
        Row4 w[kStep], a[kStep], b[kStep], r[kStep], k[kStep];
        float v[kStep][R], o[R][kStep], sum[R][kStep];
#pragma unroll
        for (int e = 0; e < kStep; ++e) {
            const int i = min(i0 + e, n - 1), t = kForward ? i : n - 1 - i;
            w[e] = row4(&s.decay[t][col]);
            a[e] = row4(&s.a[t][col]);
            b[e] = row4(&s.b[t][col]);
            r[e] = row4(&s.r[t][col]);
            if (kForward) k[e] = row4(&s.k[t][col]);
#pragma unroll
            for (int m = 0; m < R; ++m) v[e][m] = op.v != nullptr ? s.v[t][own + m] : 0.f;
        }
        if (i0 + kStep > n) {                        // tokens behind the end change nothing
#pragma unroll
            for (int e = 1; e < kStep; ++e)
                if (i0 + e >= n) {
                    w[e].lo = w[e].hi = pair(1.f, 1.f);
                    a[e] = b[e] = r[e] = none;
                    if (kForward) k[e] = none;
#pragma unroll
                    for (int m = 0; m < R; ++m) v[e][m] = 0.f;
                }
        }
#pragma unroll
        for (int e = 0; e < kStep; ++e) {            // (without branches: a token's worth of them takes as long as its sum)
            const int t = kForward ? i0 + e : n - 1 - i0 - e;
            const bool first = t >= 0 && ((starts >> t) & 1u);
            float f[R];
            if (kForward) {
#pragma unroll
                for (int m = 0; m < R; ++m) {
                    x.x[m] = keep_if(first, none, x.x[m]);
                    f[m] = dot(x.x[m], a[e]);
                }
                sum16<R>(f);
#pragma unroll
                for (int m = 0; m < R; ++m) {
                    const Pair V = pair(v[e][m], v[e][m]);
                    const Row4 kept{fma2(x.x[m].lo, w[e].lo, mul2(V, k[e].lo)), fma2(x.x[m].hi, w[e].hi, mul2(V, k[e].hi))};
                    x.x[m] = axpy(pair(f[m], f[m]), b[e], kept);
                    o[m][e] = dot(x.x[m], r[e]);
                }
                if (t == stop) x.store(out + state_at);
            } else {
                if (t == stop && t >= 0) x.add(x0 + state_at);
#pragma unroll
                for (int m = 0; m < R; ++m) {
                    x.x[m] = axpy(pair(v[e][m], v[e][m]), r[e], x.x[m]);
                    f[m] = dot(x.x[m], b[e]);
                }
                sum16<R>(f);
#pragma unroll
                for (int m = 0; m < R; ++m) {
                    const Pair S = pair(f[m], f[m]);
                    x.x[m] = keep_if(first, none, Row4{fma2(x.x[m].lo, w[e].lo, mul2(S, a[e].lo)), fma2(x.x[m].hi, w[e].hi, mul2(S, a[e].hi))});
                }
            }
#pragma unroll
            for (int m = 0; m < R; ++m) sum[m][e] = f[m];
        }
        auto pick = [l](const float* f) { return l & 2 ? (l & 1 ? f[3] : f[2]) : (l & 1 ? f[1] : f[0]); };
        const bool mine = l < kStep && i0 + l < n;   // lane l: token l of the four
        const int t = t0 + (kForward ? i0 + l : n - 1 - i0 - l);
        float q[R];
        if (kForward) {                              // lane l ends with the outputs of token l % 4
#pragma unroll
            for (int m = 0; m < R; ++m) {
                const bool odd = l & 1;
                const float even = (odd ? o[m][1] : o[m][0]) + __shfl_xor_sync(0xffffffffu, odd ? o[m][0] : o[m][1], 1);
                const float late = (odd ? o[m][3] : o[m][2]) + __shfl_xor_sync(0xffffffffu, odd ? o[m][2] : o[m][3], 1);
                q[m] = (l & 2 ? late : even) + __shfl_xor_sync(0xffffffffu, l & 2 ? even : late, 2);
            }
#pragma unroll
            for (int bit = 4; bit < 16; bit <<= 1)
#pragma unroll
                for (int m = 0; m < R; ++m) q[m] += __shfl_xor_sync(0xffffffffu, q[m], bit);
        }
        if (mine) {
#pragma unroll
            for (int m = 0; m < R; ++m) {
                if (kForward) y[at.seq + (size_t)t * at.tok + row + m] = q[m];
                if (sums != nullptr) sums[at.sum(op, t) + row + m] = pick(sum[m]);
            }
        }
    }
}

template <bool kForward, int W, int R>
__global__ void __launch_bounds__(32 * (W + 1), R == 4 ? 2 : 1)
wkv7_fp32_chain_kernel(const Operands op, const Tiles tiles, const float* __restrict__ x0, float* slots, float* sums, float* __restrict__ y,
                       float* __restrict__ out, int* __restrict__ status) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    typedef ChainSmem<W, R> Smem;
    Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
    const Place<kForward> at(op, kN / Smem::kRows);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) sm.init();
    __syncthreads();
    if (warp == W) {
        if (!fetch_chunks<kForward>(sm, op, tiles, at, slots) && status != nullptr) atomicExch(status, 7);
        return;
    }
    const int l = lane & 15, own = (warp * 2 + (lane >> 4)) * R, row = at.part * Smem::kRows + own;   // first row within the CTA, of all
    const size_t in_state = (size_t)row * kN + 4 * l, state_at = (size_t)at.bh * (kN * kN) + in_state;
    Slice<R> x;
    if (kForward) x.load(x0 + state_at); else x.clear();
    wait_for_grid_in_front();
    if (kForward && at.L == 0) x.store(out + state_at);
    bool landed = true;
    for (int it = 0; it < at.nC; ++it) {
        const int stage = it % Smem::kStages, t0 = at.chunk(it) * kC;
        landed = __all_sync(0xffffffffu, tc::mbar_wait(&sm.full[stage], (it / Smem::kStages) & 1));
        if (!landed) break;
        const int kind = sm.kind[stage];
        const typename Smem::Whole& s = sm.st[stage].whole;
        if (kForward && kind == kFresh) x.clear();
        x.store(slots + at.slot(it) + in_state);
        // (the stage of the chunk before: what was read of it went into the state that has just been stored)
        __syncwarp();
        if (it > 0 && lane == 0) tc::mbar_arrive(&sm.empty[(it - 1) % Smem::kStages]);
        if (kind != kWalked) {
            if (!kForward && at.L == t0 + kC && x0 != nullptr) x.add(x0 + state_at);
            // Slot i of a lane holds token i ^ l, so that the sums over the 16 lanes need no exchange of halves: what a lane keeps
            // at each stage are the slots without that bit, and it ends with its own token l.
            float z[R][kC];
#pragma unroll
            for (int i = 0; i < kC; ++i) {
                const Row4 left = row4(&s.left[i ^ l][4 * l]);
#pragma unroll
                for (int m = 0; m < R; ++m) z[m][i] = dot(x.x[m], left);
            }
            const Row4 p = row4(&s.decay[4 * l]);    // meanwhile: what remains of the state
#pragma unroll
            for (int m = 0; m < R; ++m) x.x[m] = mul(x.x[m], p);
#pragma unroll
            for (int bit = 8; bit > 0; bit >>= 1)
#pragma unroll
                for (int m = 0; m < R; ++m)
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (i < bit) z[m][i] += __shfl_xor_sync(0xffffffffu, z[m][i + bit], bit);
#pragma unroll
            for (int m = 0; m < R; ++m) sm.s[own + m][l] = z[m][0];
            __syncwarp();
#pragma unroll
            for (int q = 0; q < kC / 4; ++q) {       // (the terms grow towards the end that the state moves to)
                const int t = kForward ? 4 * q : kC - 4 - 4 * q;
                float4 f[R];
#pragma unroll
                for (int m = 0; m < R; ++m) f[m] = at4(&sm.s[own + m][t]);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int e = kForward ? i : 3 - i;
                    const Row4 right = row4(&s.right[t + e][4 * l]);
#pragma unroll
                    for (int m = 0; m < R; ++m) {
                        const float fe = e == 0 ? f[m].x : e == 1 ? f[m].y : e == 2 ? f[m].z : f[m].w;
                        const Pair ff = pair(fe, fe);
                        x.x[m].lo = fma2(ff, right.lo, x.x[m].lo);
                        x.x[m].hi = fma2(ff, right.hi, x.x[m].hi);
                    }
                }
            }
            x.add(&s.d[own][4 * l]);
            if (sums != nullptr) {                   // onto u, without waiting for it
                float* const sum = sums + at.sum(op, t0 + l) + row;
#pragma unroll
                for (int m = 0; m < R; ++m) atomicAdd(sum + m, z[m][0]);
            }
            if (kForward && at.L == t0 + kC) x.store(out + state_at);
            if (!kForward && kind == kFresh) x.clear();
        } else {
            walk<kForward>(x, sm.st[stage].walked, op, at, t0, sm.starts[stage], row, own, 4 * l, x0, sums, y, out);
        }
    }
    if (!kForward) {
        if (at.L == 0 && x0 != nullptr) x.add(x0 + state_at);
        x.store(out + state_at);
    }
    if (!landed && status != nullptr) atomicExch(status, 7);
}

// ------------------------------------------------------------------ the outputs --------
// y += R- S0^T for one chunk: a warp four tokens, a lane two rows of the state.
constexpr int kStatePitch = kN + 4;                  // rows 16 bytes apart in the banks: eight lanes' reads of a phase meet in none
struct OutSmem {
    float s0[kN][kStatePitch];
    float rbar[kC][kN];
};
__global__ void __launch_bounds__(128)
wkv7_fp32_outputs_kernel(const Operands op, const Tiles tiles, const float* slots, float* y) {
    __shared__ __align__(16) OutSmem sm;
    const int nC = (op.T + kC - 1) / kC, bh = blockIdx.x / nC, c = blockIdx.x % nC, bi = bh / op.H, h = bh % op.H;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, t0 = c * kC;
    const int L = min((int)op.length[bi], op.T);
    const bool flag = tid > 0 && tid < kC && t0 + tid < op.T && op.new_starts[(size_t)bi * op.T + t0 + tid] != 0;
    const bool walked = __syncthreads_or(flag) || kind_of(0, t0, op.T, L) == kWalked;
    wait_for_grid_in_front();                        // (also where there is nothing to do: see launch_in_chain)
    if (walked) return;
    const float* const state = slots + ((size_t)bh * nC + c) * (kN * kN);
    const float* const rbar = tiles.rbar + bh * tiles.head_stride + c * tiles.chunk_stride;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int at = i * 128 + tid;
        put4(&sm.s0[at >> 4][(at & 15) * 4], at4(state + at * 4));
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) put4(&sm.rbar[0][0] + (i * 128 + tid) * 4, at4(rbar + (i * 128 + tid) * 4));
    float* to = y + (size_t)bi * op.T * op.H * kN + (size_t)h * kN + (size_t)(t0 + warp * 4) * op.H * kN + lane;
    float acc[4][2];
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int m = 0; m < 2; ++m) acc[t][m] = to[(size_t)t * op.H * kN + 32 * m];
    __syncthreads();
    Pair sum[4][2];
#pragma unroll
    for (int t = 0; t < 4; ++t) sum[t][0].u = sum[t][1].u = 0;
#pragma unroll 4
    for (int j = 0; j < kN; j += 4) {
        const Row4 x0 = row4(&sm.s0[lane][j]), x1 = row4(&sm.s0[lane + 32][j]);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const Row4 g = row4(&sm.rbar[warp * 4 + t][j]);
            sum[t][0] = fma2(x0.hi, g.hi, fma2(x0.lo, g.lo, sum[t][0]));
            sum[t][1] = fma2(x1.hi, g.hi, fma2(x1.lo, g.lo, sum[t][1]));
        }
    }
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const float2 f = unpack(sum[t][m]);
            to[(size_t)t * op.H * kN + 32 * m] = acc[t][m] + (f.x + f.y);
        }
}

// ------------------------------------------------------------------ the gradients --------
// One CTA of four warps per chunk; 16 lanes have eight rows of the state as pairs of rows, a lane four columns of them.  With s and
// g known a token's step is elementwise: the forward states are rebuilt from the checkpoint (from a copy at token 8 for the second
// half) four tokens at a time and kept in registers while the state gradient comes back over them.  Sums over rows are a
// lane's own eight, then those of the eight groups, four tokens together; a sum over columns (dv) is eight shuffles.  Bound by
// shared-memory reads and the latency of eight warps per SM (255 registers): 9.8 us per chunk and SM.  Two tokens at a time: 10.9;
// eight rows by two columns per lane, which reads 1.6 times as much shared memory: 12.
constexpr int kGradThreads = 128;
constexpr int kBlk = 4;                              // tokens whose states are in registers at a time
struct GradSmem {
    float w[kC][kN], r[kC][kN], k[kC][kN], a[kC][kN], b[kC][kN], v[kC][kN], dy[kC][kN], s[kC][kN], g[kC][kN], dw[kC][kN];
    float4 mid[8][kGradThreads];                     // the state entering token 8
    float red[8][5][kBlk][kN];
    uint32_t starts;
};
__global__ void __launch_bounds__(kGradThreads, 2)
wkv7_fp32_grads_kernel(const Operands op, const float* __restrict__ vv, const float* __restrict__ ds_out, const float* __restrict__ ckpt,
                       const float* carry, const float* sums, float* __restrict__ dw, float* __restrict__ dr,
                       float* __restrict__ dk, float* dv, float* __restrict__ da, float* __restrict__ db) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    GradSmem& sm = *reinterpret_cast<GradSmem*>(smem_raw);
    const int nC = (op.T + kC - 1) / kC, bh = blockIdx.x / nC, c = blockIdx.x % nC, bi = bh / op.H, h = bh % op.H;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, t0 = c * kC;
    const int l = lane & 15, group = warp * 2 + (lane >> 4), r0 = group * 8, j0 = l * 4;
    const size_t seq = (size_t)bi * op.T * op.H * kN + (size_t)h * kN, tok = (size_t)op.H * kN;
    wait_for_grid_in_front();
    const int L = min((int)op.length[bi], op.T);
    {   // tokens behind the end change nothing: no decay, all else zero
#pragma unroll
        for (int pass = 0; pass < 2; ++pass) {
            const int t = (tid >> 4) + 8 * pass, col = l * 4;
            const bool in = t0 + t < op.T;
            const size_t at = seq + (size_t)(in ? t0 + t : 0) * tok + col;
            const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 w = at4(op.w + at), r = at4(op.r + at), k = at4(op.k + at), a = at4(op.a + at), b = at4(op.b + at), v = at4(vv + at),
                         dy = op.v != nullptr ? at4(op.v + at) : none, g = at4(dv + at), s = at4(sums + ((size_t)bh * op.T + (in ? t0 + t : 0)) * kN + col);
            const float4 e = make_float4(expf(w.x), expf(w.y), expf(w.z), expf(w.w)), d = make_float4(expf(-e.x), expf(-e.y), expf(-e.z), expf(-e.w));
            put4(&sm.w[t][col], in ? d : make_float4(1.f, 1.f, 1.f, 1.f));
            put4(&sm.dw[t][col], make_float4(-e.x * d.x, -e.y * d.y, -e.z * d.z, -e.w * d.w));
            put4(&sm.r[t][col], in ? r : none);
            put4(&sm.k[t][col], in ? k : none);
            put4(&sm.a[t][col], in ? a : none);
            put4(&sm.b[t][col], in ? b : none);
            put4(&sm.v[t][col], in ? v : none);
            put4(&sm.dy[t][col], in ? dy : none);
            put4(&sm.s[t][col], in ? s : none);
            put4(&sm.g[t][col], in ? g : none);
        }
        if (warp == 0) {
            const bool f = lane < kC && t0 + lane < op.T && op.new_starts[(size_t)bi * op.T + t0 + lane] != 0;
            const uint32_t m = __ballot_sync(0xffffffffu, f);
            if (lane == 0) sm.starts = m;
        }
    }
    const size_t tile = ((size_t)bh * nC + c) * (kN * kN) + (size_t)r0 * kN + j0;
    struct Square { Pair m[4][4]; };                 // rows r0 + 2 p, + 1; columns j0 .. j0 + 3
    auto load = [&](const float* from, size_t at) {
        Square q;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const float4 x = at4(from + at + (2 * p) * kN), z = at4(from + at + (2 * p + 1) * kN);
            q.m[p][0] = pair(x.x, z.x);
            q.m[p][1] = pair(x.y, z.y);
            q.m[p][2] = pair(x.z, z.z);
            q.m[p][3] = pair(x.w, z.w);
        }
        return q;
    };
    struct Rows { Pair m[4]; };
    auto rows = [&](const float (*of)[kN], int t) {
        Rows x;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const ulonglong2 f = *reinterpret_cast<const ulonglong2*>(&of[t][r0 + 4 * q]);
            x.m[2 * q].u = f.x;
            x.m[2 * q + 1].u = f.y;
        }
        return x;
    };
    struct Columns { Pair m[4]; };
    auto columns = [&](const float (*of)[kN], int t) {
        const float4 f = at4(&of[t][j0]);
        return Columns{{pair(f.x, f.x), pair(f.y, f.y), pair(f.z, f.z), pair(f.w, f.w)}};
    };
    Square S = load(ckpt, tile), x = load(carry, tile);
    __syncthreads();
    const uint32_t starts = sm.starts;
    auto clear = [&](Square& q) {
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int e = 0; e < 4; ++e) q.m[p][e].u = 0;
    };
    auto forward = [&](int t) {                      // S behind token t
        const Columns w = columns(sm.w, t), k = columns(sm.k, t), b = columns(sm.b, t);
        const Rows v = rows(sm.v, t), s = rows(sm.s, t);
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int e = 0; e < 4; ++e) S.m[p][e] = fma2(S.m[p][e], w.m[e], fma2(v.m[p], k.m[e], mul2(s.m[p], b.m[e])));
    };
    auto skip = [&](int from, int to) {
#pragma unroll 1
        for (int t = from; t < to; ++t) {
            if ((starts >> t) & 1u) clear(S);
            forward(t);
        }
    };
    enum { kDr, kDa, kDk, kDb, kDw };
    auto keep = [&](int which, int tt, const Pair (&x)[4]) {
        float f[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 q = unpack(x[e]);
            f[e] = q.x + q.y;
        }
        put4(&sm.red[group][which][tt][j0], make_float4(f[0], f[1], f[2], f[3]));
    };
    float* const to[5] = {dr, da, dk, db, dw};
    auto block = [&](int tb) {                       // S is the state entering token tb
        Square hist[kBlk];
#pragma unroll
        for (int tt = 0; tt < kBlk; ++tt) {
            const int t = tb + tt;
            if ((starts >> t) & 1u) clear(S);
            hist[tt] = S;
            Pair sum[4] = {{0}, {0}, {0}, {0}};
            const Rows g = rows(sm.g, t);
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
                for (int e = 0; e < 4; ++e) sum[e] = fma2(S.m[p][e], g.m[p], sum[e]);
            keep(kDa, tt, sum);
            forward(t);
            sum[0].u = sum[1].u = sum[2].u = sum[3].u = 0;
            const Rows dy = rows(sm.dy, t);
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
                for (int e = 0; e < 4; ++e) sum[e] = fma2(S.m[p][e], dy.m[p], sum[e]);
            keep(kDr, tt, sum);
        }
#pragma unroll
        for (int tt = kBlk - 1; tt >= 0; --tt) {
            const int t = tb + tt;
            if (t0 + t == L - 1 && ds_out != nullptr) {
                const Square q = load(ds_out, ((size_t)bh * kN + r0) * kN + j0);
#pragma unroll
                for (int p = 0; p < 4; ++p)
#pragma unroll
                    for (int e = 0; e < 4; ++e) x.m[p][e] = add2(x.m[p][e], q.m[p][e]);
            }
            {
                const Columns r = columns(sm.r, t);
                const Rows dy = rows(sm.dy, t);
#pragma unroll
                for (int p = 0; p < 4; ++p)
#pragma unroll
                    for (int e = 0; e < 4; ++e) x.m[p][e] = fma2(dy.m[p], r.m[e], x.m[p][e]);
            }
            Pair sum[4] = {{0}, {0}, {0}, {0}};
            {
                const Rows v = rows(sm.v, t);
#pragma unroll
                for (int p = 0; p < 4; ++p)
#pragma unroll
                    for (int e = 0; e < 4; ++e) sum[e] = fma2(x.m[p][e], v.m[p], sum[e]);
                keep(kDk, tt, sum);
            }
            sum[0].u = sum[1].u = sum[2].u = sum[3].u = 0;
            {
                const Rows s = rows(sm.s, t);
#pragma unroll
                for (int p = 0; p < 4; ++p)
#pragma unroll
                    for (int e = 0; e < 4; ++e) sum[e] = fma2(x.m[p][e], s.m[p], sum[e]);
                keep(kDb, tt, sum);
            }
            sum[0].u = sum[1].u = sum[2].u = sum[3].u = 0;
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
                for (int e = 0; e < 4; ++e) sum[e] = fma2(x.m[p][e], hist[tt].m[p][e], sum[e]);
            keep(kDw, tt, sum);
            {   // dv, the sums over the columns: eight rows, one of them left per two lanes
                const Columns k = columns(sm.k, t);
                float f[8];
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const float2 q = unpack(fma2(x.m[p][3], k.m[3], fma2(x.m[p][2], k.m[2], fma2(x.m[p][1], k.m[1], mul2(x.m[p][0], k.m[0])))));
                    f[2 * p] = q.x;
                    f[2 * p + 1] = q.y;
                }
#pragma unroll
                for (int m = 4; m > 0; m >>= 1) {
                    const bool up = lane & (2 * m);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (i < m) {
                            const float send = up ? f[i] : f[i + m], mine = up ? f[i + m] : f[i];
                            f[i] = mine + __shfl_xor_sync(0xffffffffu, send, 2 * m);
                        }
                }
                f[0] += __shfl_xor_sync(0xffffffffu, f[0], 1);
                if ((lane & 1) == 0 && t0 + t < op.T) dv[seq + (size_t)(t0 + t) * tok + r0 + (l >> 1)] = f[0];
            }
            {
                const Columns w = columns(sm.w, t), a = columns(sm.a, t);
                const Rows g = rows(sm.g, t);
#pragma unroll
                for (int p = 0; p < 4; ++p)
#pragma unroll
                    for (int e = 0; e < 4; ++e) x.m[p][e] = fma2(x.m[p][e], w.m[e], mul2(g.m[p], a.m[e]));
            }
            if ((starts >> t) & 1u) clear(x);
        }
        __syncthreads();
        const int tt = warp, j = 2 * lane;
        const size_t at = seq + (size_t)(t0 + tb + tt) * tok + j;
#pragma unroll
        for (int which = 0; which < 5; ++which) {
            float2 f = make_float2(0.f, 0.f);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const float2 x = *reinterpret_cast<const float2*>(&sm.red[q][which][tt][j]);
                f.x += x.x;
                f.y += x.y;
            }
            if (which == kDw) {
                const float2 x = *reinterpret_cast<const float2*>(&sm.dw[tb + tt][j]);
                f.x *= x.x;
                f.y *= x.y;
            }
            if (t0 + tb + tt < op.T) *reinterpret_cast<float2*>(to[which] + at) = f;
        }
        __syncthreads();
    };
    skip(0, 8);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float2 lo = unpack(S.m[i >> 1][2 * (i & 1)]), hi = unpack(S.m[i >> 1][2 * (i & 1) + 1]);
        sm.mid[i][tid] = make_float4(lo.x, lo.y, hi.x, hi.y);
    }
#pragma unroll 1
    for (int tb = kC - kBlk; tb >= 0; tb -= kBlk) {
        if (tb == 8) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 f = sm.mid[i][tid];
                S.m[i >> 1][2 * (i & 1)] = pair(f.x, f.y);
                S.m[i >> 1][2 * (i & 1) + 1] = pair(f.z, f.w);
            }
        } else if (tb < 8) {
            S = load(ckpt, tile);
        }
        if (tb & 4) skip(tb - 4, tb);
        block(tb);
    }
}

// ------------------------------------------------------------------ launchers --------
constexpr int kTileFloats = 3 * kTile + kN;          // W~, b^, R-, P_C of a chunk in a workspace
int chunks_of(int T) { return (T + kC - 1) / kC; }

template <typename K>
bool opted_in(K kern, int smem, DeviceOnce& once) {
    return once.ok([kern, smem]() { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); });
}
template <bool kForward>
int launch_prepare(cudaStream_t st, int heads, const Operands& op, const Tiles& tiles, float* slots, float* sums, float* y) {
    auto kern = wkv7_fp32_prepare_kernel<kForward>;
    static DeviceOnce once;
    if (!opted_in(kern, (int)sizeof(PrepSmem), once)) return B200WKV_ELAUNCH;
    kern<<<heads * chunks_of(op.T), kPrepThreads, sizeof(PrepSmem), st>>>(op, tiles, slots, sums, y);
    return cudaGetLastError() == cudaSuccess ? B200WKV_OK : B200WKV_ELAUNCH;
}
template <bool kForward, int W, int R>
int launch_chain_split(cudaStream_t st, int heads, const Operands& op, const Tiles& tiles, const float* x0, float* slots, float* sums, float* y, float* out) {
    auto kern = wkv7_fp32_chain_kernel<kForward, W, R>;
    typedef ChainSmem<W, R> Smem;
    static DeviceOnce once;
    if (!opted_in(kern, (int)sizeof(Smem), once)) return B200WKV_ELAUNCH;
    return launch_behind(kern, heads * (kN / Smem::kRows), 32 * (W + 1), sizeof(Smem), st, op, tiles, x0, slots, sums, y, out,
                         wkv7_chunk_status_word()) == cudaSuccess ? B200WKV_OK : B200WKV_ELAUNCH;
}
// As few rows per lane as leave every CTA an SM.  Measured (us, forward chain): 8 heads, T = 256: 13.2 with W, R = 2, 1, 16.6 with
// 4, 2, 19.8 with 4, 4; 24 heads, T = 512: 47, 30, 36; 48 heads: 44 with 4, 2, 43 with 4, 4; 128 heads: 79 and 58.
template <bool kForward, typename... A>
int launch_chain(cudaStream_t st, int heads, A... args) {
    const int sms = sm_count_of_current_device();
    if (16 * heads <= sms) return launch_chain_split<kForward, 2, 1>(st, heads, args...);
    if (8 * heads <= sms) return launch_chain_split<kForward, 4, 1>(st, heads, args...);
    if (4 * heads <= sms) return launch_chain_split<kForward, 4, 2>(st, heads, args...);
    return launch_chain_split<kForward, 4, 4>(st, heads, args...);
}
}  // namespace

// Whether calls with gradients take these kernels (the rest of wkv7_chain.cu and wkv7_seq.cu: fewer tokens, and residuals without
// their room).  The device is faster here at every size measured; the line is a host's.  An eager forward and backward takes the host of
// a B200 some 105 us with the kernels there and 112 with the four more here, so that below the line, where those kernels are done
// by then, these cost 6 us.  Calls from a captured graph, which have no such floor, would gain from fewer tokens on.  us, there / here, eager (graph):
// 8 heads, T=192 105 / 112 (70 / 49), 256 106 / 113 (84 / 54), 320 127 / 112 (119 / 67); 24 heads, 96 106 / 113 (57 / 46), 160 108 / 113
// (94 / 59), 208 135 / 114 (127 / 80); 40 heads, 104 107 / 113 (86 / 62), 160 130 / 113 (123 / 82); 64 heads, 64 106 / 112 (72 / 54), 104 116 / 111
// (107 / 85); 160 heads, 64 178 / 122; 640 heads, 64 534 / 395.  With a flag every 16 tokens, eager: 8 heads, T=1024 330 / 303; 24 heads, 208
// 142 / 125, 2048 1104 / 861; 160 heads, 64 179 / 144.
bool wkv7_fp32_takes(int B, int T, int H) { return chunks_of(T) >= 4 && chunks_of(T) * ((long long)B * H + 16) >= 440; }

// What a forward call without a residual wants as a workspace (0: it takes the token-by-token chain).  That chain takes the same
// time up to a head per SM and doesn't mind flags, this one shares the device with what is done beside it, and a flagged or cut chunk
// is walked: up to a quarter of a head per SM, and from 13 chunks on, where no count of heads loses at a flag every 256 tokens and
// lengths of T / 2 to T.  us, that chain / here, without flags, and with those flags and lengths:
//     4 heads:   T=144 21 / 17, 21 / 21    208 27 / 20, 27 / 23    512 60 / 31, 60 / 37    2000 223 / 97, 224 / 109
//     16 heads:  T=160 23 / 21, 23 / 27    208 27 / 24, 27 / 27    512 60 / 45, 61 / 52    2000 224 / 146, 224 / 166
//     24 heads:  T=160 27 / 23, 27 / 27    208 34 / 27, 35 / 31    512 76 / 52, 77 / 56    2000 282 / 179, 288 / 199
//     36 heads:  T=176 29 / 27, 31 / 33    208 35 / 33, 35 / 33    512 76 / 60, 77 / 67    2000 282 / 220, 287 / 242
//     48 heads:  T=208 41 / 37, 41 / 42    512 92 / 78, 93 / 99    64 heads:  T=512 92 / 92, 93 / 111
// With a flag every 64 tokens they are equal at T=256 to 512 (4 heads 33 / 33, 36 heads 82 / 82) and these faster behind that (4 heads, T=2000
// 225 / 138).  Every 16 tokens 4 heads take 33 / 49 at T=256 and 230 / 230 at 2000, 24 heads 48 / 60 and 330 / 325: the host doesn't know
// the flags.  The last limit bounds the workspace, 2 GiB.
size_t wkv7_fp32_workspace_bytes(int B, int T, int H) {
    if (chunks_of(T) < 13 || 4 * (long long)B * H > sm_count_of_current_device()) return 0;
    const size_t bytes = (size_t)B * H * chunks_of(T) * (kN * kN + kTileFloats) * sizeof(float);
    return bytes <= ((size_t)2 << 30) ? bytes : 0;
}
// What a forward leaves for its backward: the checkpoints and s of every token.  Besides, both want as much room as the checkpoints
// have while they run (the forward for its tiles, the backward for the state gradients between the chunks): a workspace of each, or
// the residual's middle.
size_t wkv7_fp32_state_bytes(int B, int T, int H) { return (size_t)B * H * chunks_of(T) * kN * kN * sizeof(float); }
size_t wkv7_fp32_kept_bytes(int B, int T, int H) { return wkv7_fp32_state_bytes(B, T, H) + (size_t)B * H * T * kN * sizeof(float); }

int wkv7_fp32_fwd(cudaStream_t st, int B, int T, int H, const void* w, const void* r, const void* k, const void* v, const void* a,
                  const void* b, const void* s0, const uint32_t* length, const uint8_t* ns, void* y, void* s_out, void* residual,
                  size_t residual_bytes, void* workspace) {
    const int heads = B * H, nC = chunks_of(T);
    const Operands op{T, H, (const float*)w, (const float*)r, (const float*)k, (const float*)v, (const float*)a, (const float*)b, length, ns};
    const size_t states = (size_t)heads * nC * kN * kN, stride = residual != nullptr ? (size_t)kN * kN : (size_t)kTileFloats;
    const bool room = residual != nullptr && residual_bytes >= wkv7_fp32_kept_bytes(B, T, H) + wkv7_fp32_state_bytes(B, T, H);
    float* const slots = (float*)(residual != nullptr ? residual : workspace);
    float* const base = residual == nullptr || room ? slots + states : (float*)workspace;
    float* const sums = residual == nullptr ? nullptr : room ? base + states : slots + states;
    const Tiles tiles{base, base + kTile, base + 2 * kTile, base + 3 * kTile, stride * nC, stride};
    int s = launch_prepare<true>(st, heads, op, tiles, slots, sums, (float*)y);
    if (s != B200WKV_OK) return s;
    s = launch_chain<true>(st, heads, op, tiles, (const float*)s0, slots, sums, (float*)y, (float*)s_out);
    if (s != B200WKV_OK) return s;
    return launch_behind(wkv7_fp32_outputs_kernel, heads * nC, 128, 0, st, op, tiles, slots, (float*)y) == cudaSuccess ? B200WKV_OK : B200WKV_ELAUNCH;
}

// The tiles of the chain lie in the buffers of the gradients, as [head][token][64], until the last kernel writes these; g lies in
// dv's, where the last kernel's CTAs write over their own.
int wkv7_fp32_bwd(cudaStream_t st, int B, int T, int H, const void* w, const void* r, const void* k, const void* v, const void* a,
                  const void* b, const uint32_t* length, const uint8_t* ns, const void* dy, const void* ds_out, void* residual,
                  size_t residual_bytes, void* workspace, void* dw, void* dr, void* dk, void* dv, void* da, void* db, void* ds0) {
    const int heads = B * H, nC = chunks_of(T);
    const Operands op{T, H, (const float*)w, (const float*)r, (const float*)k, (const float*)dy, (const float*)a, (const float*)b, length, ns};
    const size_t states = (size_t)heads * nC * kN * kN;
    const bool room = residual_bytes >= wkv7_fp32_kept_bytes(B, T, H) + wkv7_fp32_state_bytes(B, T, H);
    float *const ckpt = (float*)residual, *const carry = room ? ckpt + states : (float*)workspace, *const sums = ckpt + (room ? 2 : 1) * states;
    const Tiles tiles{(float*)dk, (float*)da, nullptr, (float*)dw, (size_t)T * kN, (size_t)kTile};
    int s = launch_prepare<false>(st, heads, op, tiles, carry, (float*)dv, nullptr);
    if (s != B200WKV_OK) return s;
    s = launch_chain<false>(st, heads, op, tiles, (const float*)ds_out, carry, (float*)dv, nullptr, (float*)ds0);
    if (s != B200WKV_OK) return s;
    auto kern = wkv7_fp32_grads_kernel;
    static DeviceOnce once;
    if (!opted_in(kern, (int)sizeof(GradSmem), once)) return B200WKV_ELAUNCH;
    return launch_behind(kern, heads * nC, kGradThreads, sizeof(GradSmem), st, op, (const float*)v, (const float*)ds_out, ckpt, carry, sums, (float*)dw, (float*)dr,
                         (float*)dk, (float*)dv, (float*)da, (float*)db) == cudaSuccess ? B200WKV_OK : B200WKV_ELAUNCH;
}

}  // namespace b200wkv
