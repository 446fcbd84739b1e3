// Token shift with start flags and the carried last row: the per-token state that the callers of the
// WKV operator maintain next to it (jaxrwkv src/jaxrwkv/rwkv7.py:226-235 and :254 for time mixing,
// :192-197 for channel mixing).  For every mix m:
//   shifted[t] = new_starts[t] ? 0 : (t == 0 ? prev : x[t-1])
//   out_m[t]   = x[t] + (shifted[t] - x[t]) * mix_m
//   state_out  = x[(length - 1) mod T]            (the reference indexes x[length-1]; length 0 wraps)
// One pass over x, M outputs: purely HBM-bound, so every thread moves V channels per access with
// V = 16 bytes / element size when the channel count allows it (else V = 4).
#include "common.cuh"
#include "device_once.cuh"
#include "host_calls.h"

namespace b200wkv {
namespace {

template <int V> struct Vec { float f[V]; };
struct MixPtrs { const void* p[8]; };   // one row of D coefficients each

template <int V, typename T> __device__ __forceinline__ Vec<V> loadv(const T* p);
template <> __device__ __forceinline__ Vec<4> loadv<4, float>(const float* p) {
    const float4 q = load4(p);
    return Vec<4>{{q.x, q.y, q.z, q.w}};
}
template <> __device__ __forceinline__ Vec<4> loadv<4, __nv_bfloat16>(const __nv_bfloat16* p) {
    const float4 q = load4(p);
    return Vec<4>{{q.x, q.y, q.z, q.w}};
}
template <> __device__ __forceinline__ Vec<8> loadv<8, __nv_bfloat16>(const __nv_bfloat16* p) {
    const uint4 raw = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
    Vec<8> r;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 t = __bfloat1622float2(h[i]);
        r.f[2 * i] = t.x;
        r.f[2 * i + 1] = t.y;
    }
    return r;
}
__device__ __forceinline__ void storev(float* p, const Vec<4>& v) { store4(p, make_float4(v.f[0], v.f[1], v.f[2], v.f[3])); }
__device__ __forceinline__ void storev(__nv_bfloat16* p, const Vec<4>& v) {
    store4(p, make_float4(v.f[0], v.f[1], v.f[2], v.f[3]));
}
__device__ __forceinline__ void storev(__nv_bfloat16* p, const Vec<8>& v) {
    uint4 raw;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v.f[2 * i], v.f[2 * i + 1]);
    *reinterpret_cast<uint4*>(p) = raw;
}
// V channels as they lie in memory (16 or 8 bytes): what a thread keeps of a load until it uses it
template <int V, typename T> struct RawVec;
template <> struct RawVec<4, float> {
    float4 q;
    __device__ __forceinline__ void load(const float* p) { q = *reinterpret_cast<const float4*>(p); }
    __device__ __forceinline__ Vec<4> get() const { return Vec<4>{{q.x, q.y, q.z, q.w}}; }
};
template <> struct RawVec<4, __nv_bfloat16> {
    uint2 q;
    __device__ __forceinline__ void load(const __nv_bfloat16* p) { q = *reinterpret_cast<const uint2*>(p); }
    __device__ __forceinline__ Vec<4> get() const {
        return Vec<4>{{__uint_as_float(q.x << 16), __uint_as_float(q.x & 0xffff0000u), __uint_as_float(q.y << 16),
                       __uint_as_float(q.y & 0xffff0000u)}};
    }
};
template <> struct RawVec<8, __nv_bfloat16> {
    uint4 q;
    __device__ __forceinline__ void load(const __nv_bfloat16* p) { q = *reinterpret_cast<const uint4*>(p); }
    __device__ __forceinline__ Vec<8> get() const {
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
        Vec<8> r;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            r.f[2 * i] = __uint_as_float(w[i] << 16);
            r.f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
        return r;
    }
};

template <int V> __device__ __forceinline__ Vec<V> zerov() {
    Vec<V> r;
#pragma unroll
    for (int i = 0; i < V; ++i) r.f[i] = 0.f;
    return r;
}

__device__ __forceinline__ int last_row(uint32_t length, int Tlen) {
    const int L = (int)min(length, (uint32_t)0x7fffffff);
    return ((L - 1) % Tlen + Tlen) % Tlen;
}

// grid (B*T, ceil(D / V / 128)); one token row per blockIdx.x
template <typename T, int V>
__global__ void token_shift_fwd_kernel(int B, int Tlen, int D, int M, const T* __restrict__ x, const T* __restrict__ prev,
                                       const MixPtrs mix, const uint32_t* __restrict__ length,
                                       const uint8_t* __restrict__ new_starts, T* __restrict__ out,
                                       T* __restrict__ state_out) {
    const int d = (blockIdx.y * blockDim.x + threadIdx.x) * V;
    const int bt = blockIdx.x;
    if (d >= D) return;
    const int bi = bt / Tlen, t = bt % Tlen;
    const size_t row = (size_t)bt * D + d;
    const Vec<V> xc = loadv<V>(x + row);
    Vec<V> df = zerov<V>();
    if (!new_starts[bt]) df = (t == 0) ? loadv<V>(prev + (size_t)bi * D + d) : loadv<V>(x + row - D);
#pragma unroll
    for (int i = 0; i < V; ++i) df.f[i] -= xc.f[i];
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        if (m >= M) break;
        const Vec<V> c = loadv<V>((const T*)mix.p[m] + d);
        Vec<V> o;
#pragma unroll
        for (int i = 0; i < V; ++i) o.f[i] = fmaf(df.f[i], c.f[i], xc.f[i]);
        storev(out + ((size_t)m * B * Tlen + bt) * D + d, o);
    }
    if (t == last_row(length[bi], Tlen)) storev(state_out + (size_t)bi * D + d, xc);
}

// Backward.  A thread owns V channels of a tile of B200WKV_SHIFT_TILE tokens of one batch row, or of one of the kParts parts
// of it, and walks its tokens from the last to the first (the loads do not depend on the walk, so they pipeline; a part reads
// the token behind it for itself).
// The mix gradients leave as one fp32 partial sum per (batch row, tile): deterministic, no atomics.
//   gx[t] = sum_m g_m[t] (1 - c_m) + [t+1 < T and not start[t+1]] sum_m g_m[t+1] c_m + [t == last] gstate
// grid (ceil(D / V / kLanes), tiles, B)
// Tokens are taken G at a time: the G x (MM + 1) loads of a group are all issued, in packed form, before the first token of the group
// is worked on.  kThreads per SM, which bounds the registers (0: 255).
template <typename T, int V, int MM, int kLanes, int kParts, int G, int kThreads>
__global__ void __launch_bounds__(kLanes * kParts, kThreads / (kLanes * kParts))
token_shift_bwd_kernel(int B, int Tlen, int D, const T* __restrict__ x, const T* __restrict__ prev,
                       const MixPtrs mix, const uint32_t* __restrict__ length,
                       const uint8_t* __restrict__ new_starts, const T* __restrict__ gout,
                       const T* __restrict__ gstate, T* __restrict__ gx, T* __restrict__ gprev,
                       float* __restrict__ gmix) {
    const int lane = threadIdx.x % kLanes, part = threadIdx.x / kLanes;
    const int d = (blockIdx.x * kLanes + lane) * V;
    const int tile = blockIdx.y, ntile = gridDim.y;
    const int bi = blockIdx.z;
    if (kParts == 1 && d >= D) return;
    // this thread's tokens (none, where the part lies behind the sequence's end or the channels behind the last)
    const int t0 = tile * B200WKV_SHIFT_TILE + part * (B200WKV_SHIFT_TILE / kParts);
    const int t1 = kParts == 1 || d < D ? min(Tlen, t0 + B200WKV_SHIFT_TILE / kParts) : t0;
    const bool any = kParts == 1 || t0 < t1;
    __shared__ float sums[kParts > 1 ? kParts - 1 : 1][MM][V][kLanes];
    static_assert(B200WKV_SHIFT_TILE % kParts == 0, "parts of whole tokens");
    const int last = last_row(length[bi], Tlen);
    RawVec<V, T> craw[MM];   // the mix coefficients stay packed; unpacking them at each use is cheaper than the registers
    Vec<V> acc[MM];
#pragma unroll
    for (int m = 0; m < MM; ++m) {
        if (any) craw[m].load((const T*)mix.p[m] + d);
        acc[m] = zerov<V>();
    }
    const size_t base = (size_t)bi * Tlen * D + d;
    const size_t mstride = (size_t)B * Tlen * D;
    const uint8_t* ns = new_starts + (size_t)bi * Tlen;
    Vec<V> carry = zerov<V>();   // what token t+1 hands back to token t
    if (any && t1 < Tlen && !ns[t1]) {
#pragma unroll
        for (int m = 0; m < MM; ++m) {
            const Vec<V> g = loadv<V>(gout + m * mstride + base + (size_t)t1 * D);
            const Vec<V> cm = craw[m].get();
#pragma unroll
            for (int i = 0; i < V; ++i) carry.f[i] = fmaf(g.f[i], cm.f[i], carry.f[i]);
        }
    }
    Vec<V> xc = zerov<V>();
    if (any) xc = loadv<V>(x + base + (size_t)(t1 - 1) * D);
    for (int tg = t1 - 1; tg >= t0; tg -= G) {
        RawVec<V, T> rg[G][MM], rx[G];
#pragma unroll
        for (int j = 0; j < G; ++j) {
            const int t = tg - j;
            if (t >= t0) {
#pragma unroll
                for (int m = 0; m < MM; ++m) rg[j][m].load(gout + m * mstride + base + (size_t)t * D);
                // the row before: needed as this token's shift and as the next token's x
                rx[j].load(t > 0 ? x + base + (size_t)(t - 1) * D : prev + (size_t)bi * D + d);
            }
        }
#pragma unroll
        for (int j = 0; j < G; ++j) {
            const int t = tg - j;
            if (t < t0) break;
            const bool st = ns[t] != 0;
            const Vec<V> xp = rx[j].get();
            Vec<V> keep = zerov<V>(), pass = zerov<V>(), df;
#pragma unroll
            for (int i = 0; i < V; ++i) df.f[i] = (st ? 0.f : xp.f[i]) - xc.f[i];
#pragma unroll
            for (int m = 0; m < MM; ++m) {
                const Vec<V> g = rg[j][m].get();
                const Vec<V> cm = craw[m].get();
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    keep.f[i] = fmaf(g.f[i], 1.f - cm.f[i], keep.f[i]);
                    pass.f[i] = fmaf(g.f[i], cm.f[i], pass.f[i]);
                    acc[m].f[i] = fmaf(g.f[i], df.f[i], acc[m].f[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < V; ++i) keep.f[i] += carry.f[i];
            if (t == last && gstate != nullptr) {
                const Vec<V> gs = loadv<V>(gstate + (size_t)bi * D + d);
#pragma unroll
                for (int i = 0; i < V; ++i) keep.f[i] += gs.f[i];
            }
            storev(gx + base + (size_t)t * D, keep);
#pragma unroll
            for (int i = 0; i < V; ++i) carry.f[i] = st ? 0.f : pass.f[i];
            xc = xp;
        }
    }
    if (any && t0 == 0) storev(gprev + (size_t)bi * D + d, carry);
    // the parts' sums meet in a fixed order
    if (part > 0) {
#pragma unroll
        for (int m = 0; m < MM; ++m)
#pragma unroll
            for (int i = 0; i < V; ++i) sums[part - 1][m][i][lane] = acc[m].f[i];
    }
    if (kParts > 1) __syncthreads();
    if (kParts > 1 && (part > 0 || d >= D)) return;
#pragma unroll
    for (int m = 0; m < MM; ++m)
#pragma unroll
        for (int p = 0; p < kParts - 1; ++p)
#pragma unroll
            for (int i = 0; i < V; ++i) acc[m].f[i] += sums[p][m][i][lane];
#pragma unroll
    for (int m = 0; m < MM; ++m) {
        float* dst = gmix + (((size_t)bi * ntile + tile) * MM + m) * D + d;
#pragma unroll
        for (int i = 0; i < V; i += 4) store4(dst + i, make_float4(acc[m].f[i], acc[m].f[i + 1], acc[m].f[i + 2], acc[m].f[i + 3]));
    }
}

template <typename T, int V>
void launch_fwd(cudaStream_t st, int B, int Tlen, int D, int M, const void* x, const void* prev, const MixPtrs& mix,
                const uint32_t* length, const uint8_t* ns, void* out, void* state_out) {
    dim3 grid(B * Tlen, (D / V + 127) / 128);
    token_shift_fwd_kernel<T, V><<<grid, 128, 0, st>>>(B, Tlen, D, M, (const T*)x, (const T*)prev, mix, length, ns,
                                                       (T*)out, (T*)state_out);
}

template <typename T, int V, int MM>
void launch_bwd_m(cudaStream_t st, int B, int Tlen, int D, const void* x, const void* prev, const MixPtrs& mix,
                  const uint32_t* length, const uint8_t* ns, const void* gout, const void* gstate, void* gx, void* gprev,
                  void* gmix) {
    const int tiles = (Tlen + B200WKV_SHIFT_TILE - 1) / B200WKV_SHIFT_TILE;
    auto launch = [&](auto kernel, int lanes, int parts, int channels = V) {
        const dim3 grid((D / channels + lanes - 1) / lanes, tiles, B);
        kernel<<<grid, lanes * parts, 0, st>>>(B, Tlen, D, (const T*)x, (const T*)prev, mix, length, ns, (const T*)gout, (const T*)gstate, (T*)gx,
                                               (T*)gprev, (float*)gmix);
    };
    const long long sms = sm_count_of_current_device();
    auto fits = [&](int lanes, int per_sm) { return (long long)((D / V + lanes - 1) / lanes) * tiles * B <= per_sm * sms; };
    if constexpr (sizeof(T) == 4) {
        // Fewer blocks than SMs: four parts per tile instead, of 32 x V channels.  With more, whole tiles keep more of a row together.
        if (fits(64, 1)) launch(token_shift_bwd_kernel<T, V, MM, 32, 4, 4, 0>, 32, 4);
        else launch(token_shift_bwd_kernel<T, V, MM, 64, 1, 4, 0>, 64, 1);
    } else {
        // A thread's walk is a chain of groups, 2.7 us each, and what hides it is what is in flight besides: threads with four channels
        // (with eight, 255 registers held groups of four tokens), and of the splits the finest whose blocks are all resident at once;
        // once that is many threads anyway, they need less in flight each.  us, eight channels (whole tiles or four parts) / here, M=6:
        //   D=768   T=256  B=1  15 / 8.3    T=512  B=8 28 / 16.5                   D=2048  T=831  B=1  20 / 14
        //   D=2048  T=1024 B=2  32 / 20 by 64 lanes, 2 parts of groups of 8 (23 by 32 lanes and 4 parts, which do not fit at once)
        //   D=2048  T=1000 B=3  49 / 27 by 2 parts, groups of 4 (8: 32)
        //   D=2048  T=1024 B=4  52 / 35 by whole tiles, groups of 8 (42 by 2 parts)
        //   D=768   T=2048 B=8  63 / 43, groups of 5 (8: 58, 3: 49)
        //   D=2048  T=1024 B=8  73 / 57, groups of 3 (5: 70)    T=4096 B=8 234 / 200
        // Fewer rows of mix leave registers for more threads and longer groups, and with what six rows take they have too little in flight
        // (one row, D=2048, T=4096, B=8: 92).  us as above, M=1, 2, 3, 4 (two rows of 9-12 blocks per SM: by eight channels):
        //   D=2048  T=1024 B=2  11 / 10.4   12.8 / 12.4   14.4 / 14.4   16.5 / 16.5        B=4  25 / 15   28 / 18   31 / 23   35 / 27
        //   D=768   T=2048 B=8  29 / 23   33 / 27   39 / 31   42 / 33
        //   D=2048  T=1024 B=8  31 / 25   35 / 30   41 / 35   45 / 41     B=16 41 / 41   68 / 55   75 / 65   83 / 77
        //   D=2048  T=4096 B=8  76 / 76   107 / 99   143 / 119   157 / 143
        if constexpr (MM >= 5) {
            if (fits(32, 3)) launch(token_shift_bwd_kernel<T, V, MM, 32, 4, 4, 384>, 32, 4);
            else if (fits(64, 2)) launch(token_shift_bwd_kernel<T, V, MM, 64, 2, 8, 256>, 64, 2);
            else if (fits(64, 3)) launch(token_shift_bwd_kernel<T, V, MM, 64, 2, 4, 384>, 64, 2);
            else if (fits(64, 4)) launch(token_shift_bwd_kernel<T, V, MM, 64, 1, 8, 256>, 64, 1);
            else if (fits(64, 6)) launch(token_shift_bwd_kernel<T, V, MM, 64, 1, 5, 384>, 64, 1);
            else launch(token_shift_bwd_kernel<T, V, MM, 64, 1, 3, 512>, 64, 1);
        } else if constexpr (MM >= 3) {
            if (fits(32, 4)) launch(token_shift_bwd_kernel<T, V, MM, 32, 4, 4, 512>, 32, 4);
            else if (fits(64, 3)) launch(token_shift_bwd_kernel<T, V, MM, 64, 2, 4, 384>, 64, 2);
            else if (fits(64, 4)) launch(token_shift_bwd_kernel<T, V, MM, 64, 2, 4, 512>, 64, 2);
            else if (fits(64, 6)) launch(token_shift_bwd_kernel<T, V, MM, 64, 1, 8, 384>, 64, 1);
            else launch(token_shift_bwd_kernel<T, V, MM, 64, 1, MM == 3 ? 6 : 4, 512>, 64, 1);
        } else {
            if (fits(32, MM == 1 ? 6 : 4)) launch(token_shift_bwd_kernel<T, V, MM, 32, 4, 4, MM == 1 ? 768 : 512>, 32, 4);
            else if (fits(64, 4)) launch(token_shift_bwd_kernel<T, V, MM, 64, 2, 8, 512>, 64, 2);
            else if (fits(64, 8)) launch(token_shift_bwd_kernel<T, V, MM, 64, 1, 8, 512>, 64, 1);
            else if (MM == 2 && fits(64, 12) && D % 8 == 0) launch(token_shift_bwd_kernel<T, 8, 2, 64, 1, 4, 0>, 64, 1, 8);
            else if (fits(64, 12)) launch(token_shift_bwd_kernel<T, V, MM, 64, 1, 4, 768>, 64, 1);
            else launch(token_shift_bwd_kernel<T, V, MM, 64, 1, MM == 1 ? 4 : 8, MM == 1 ? 1024 : 512>, 64, 1);
        }
    }
}

template <typename T, int V>
void launch_bwd(cudaStream_t st, int B, int Tlen, int D, int M, const void* x, const void* prev, const MixPtrs& mix,
                const uint32_t* length, const uint8_t* ns, const void* gout, const void* gstate, void* gx, void* gprev,
                void* gmix) {
#define B200WKV_SHIFT_CASE(MM) \
    case MM: launch_bwd_m<T, V, MM>(st, B, Tlen, D, x, prev, mix, length, ns, gout, gstate, gx, gprev, gmix); break;
    switch (M) {
        B200WKV_SHIFT_CASE(1) B200WKV_SHIFT_CASE(2) B200WKV_SHIFT_CASE(3) B200WKV_SHIFT_CASE(4)
        B200WKV_SHIFT_CASE(5) B200WKV_SHIFT_CASE(6) B200WKV_SHIFT_CASE(7) B200WKV_SHIFT_CASE(8)
    }
#undef B200WKV_SHIFT_CASE
}
}  // namespace

int token_shift_fwd(cudaStream_t st, int dtype, int B, int T, int D, int M, const void* x, const void* prev,
                    const void* const* mix, const uint32_t* length, const uint8_t* ns, void* out, void* state_out) {
    MixPtrs rows;
    for (int m = 0; m < 8; ++m) rows.p[m] = mix[m < M ? m : 0];
    if (dtype == B200WKV_F32) launch_fwd<float, 4>(st, B, T, D, M, x, prev, rows, length, ns, out, state_out);
    else if (D % 8 == 0) launch_fwd<__nv_bfloat16, 8>(st, B, T, D, M, x, prev, rows, length, ns, out, state_out);
    else launch_fwd<__nv_bfloat16, 4>(st, B, T, D, M, x, prev, rows, length, ns, out, state_out);
    return cudaGetLastError() == cudaSuccess ? B200WKV_OK : B200WKV_ELAUNCH;
}

int token_shift_bwd(cudaStream_t st, int dtype, int B, int T, int D, int M, const void* x, const void* prev,
                    const void* const* mix, const uint32_t* length, const uint8_t* ns, const void* gout, const void* gstate,
                    void* gx, void* gprev, void* gmix) {
    MixPtrs rows;
    for (int m = 0; m < 8; ++m) rows.p[m] = mix[m < M ? m : 0];
    if (dtype == B200WKV_F32) launch_bwd<float, 4>(st, B, T, D, M, x, prev, rows, length, ns, gout, gstate, gx, gprev, gmix);
    else launch_bwd<__nv_bfloat16, 4>(st, B, T, D, M, x, prev, rows, length, ns, gout, gstate, gx, gprev, gmix);
    return cudaGetLastError() == cudaSuccess ? B200WKV_OK : B200WKV_ELAUNCH;
}

}  // namespace b200wkv
