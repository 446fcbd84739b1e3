// RWKV-7, fp32 arithmetic: the two recurrences that are sequential in time, split over rows of the state.
//
// Forward and state-gradient recurrence have the same form, row by row of the 64x64 state:
//   forward, t ascending:   s = x . a_t;                  x <- x w_t + V k_t + s b_t;   y_t = x . r_t    (V = v_t[row])
//   backward, t descending: x <- x + V r_t;  s = x . b_t; x <- x w_t + s a_t                             (V = dy_t[row])
// (jaxrwkv src/jaxrwkv/rwkv7.py:199-220 and its reverse).  Rows never meet, so a (sequence, head) is spread over CTAs of 8 R
// rows: two computing warps, eight lanes to R rows, eight columns of each row in a lane.  R trades latency for throughput:
// a token's vectors are read from shared memory once for R rows, and a read costs its full width per lane even where lanes
// get the same words, while one warp needs two cycles per multiply-add of its own.  See rows_per_lane() for the choice.
// Streaming warps stage the next chunk, with the decay's exponentials taken.
// B*H = 24, T = 512, fp32: forward 227 us with a row per thread and one CTA per head (850 cycles per token), 76 us now.
#include "common.cuh"
#include "device_once.cuh"
#include "wkv7_exact.cuh"

namespace b200wkv {
namespace {

constexpr int kCompute = 64;
constexpr int kStream = 128;
constexpr int kThreads = kCompute + kStream;

template <int R>
struct ChainSmem {
    static constexpr int kRows = 8 * R;    // of a CTA
    float vec[2][5][kExactChunk][kN];      // w, a, b, k (forward only), r
    float rows[2][kExactChunk][kRows];     // v or dy
    float y[2][kExactChunk][kRows];
    uint32_t starts[2];                    // bit per token of the chunk
};
enum { kW, kA, kB, kK, kR };
struct Plain { static constexpr bool value = true; };
struct Marked { static constexpr bool value = false; };

// a lane's eight columns of a row: 4 p + 32 q .. + 3 for q = 0, 1, so that the eight lanes' loads are 128 contiguous bytes
struct Cols { Pair v[4]; };
__device__ __forceinline__ Cols cols(const float* row, int p) {
    Cols c;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(row + 32 * q + 4 * p);
        c.v[2 * q].u = u.x;
        c.v[2 * q + 1].u = u.y;
    }
    return c;
}
template <typename T>
__device__ __forceinline__ Cols load_cols(const T* row, int p) {
    Cols c;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const float4 f = load4(row + 32 * q + 4 * p);
        c.v[2 * q] = pair(f.x, f.y);
        c.v[2 * q + 1] = pair(f.z, f.w);
    }
    return c;
}
template <typename T>
__device__ __forceinline__ void store_cols(T* row, int p, const Cols& c) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const float2 a = unpack(c.v[2 * q]), b = unpack(c.v[2 * q + 1]);
        store4(row + 32 * q + 4 * p, make_float4(a.x, a.y, b.x, b.y));
    }
}
__device__ __forceinline__ float dot(const Cols& a, const Cols& b) {
    const Pair e = fma2(a.v[2], b.v[2], mul2(a.v[0], b.v[0])), o = fma2(a.v[3], b.v[3], mul2(a.v[1], b.v[1]));
    const float2 s = unpack(add2(e, o));
    return s.x + s.y;
}

__device__ __forceinline__ float sum8(float x) {   // over the eight lanes of a row
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    x += __shfl_xor_sync(0xffffffffu, x, 2);
    x += __shfl_xor_sync(0xffffffffu, x, 4);
    return x;
}
// v[i] summed over the eight lanes, the sum of v[lane % 8] returned: seven shuffles for eight sums
__device__ __forceinline__ float transpose_sum8(float* v, int lane) {
#pragma unroll
    for (int m = 4; m > 0; m >>= 1) {
        const bool up = lane & m;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i < m) {
                const float send = up ? v[i] : v[i + m], keep = up ? v[i + m] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
            }
    }
    return v[0];
}

// Forward: writes y, out = s_out and, where wanted, the state entering every chunk (ckpt).  Backward (kForward false): v is
// dy (NULL: zero), x0 the returned state's cotangent (NULL: zero), out is ds0, k and y are not used, and `ckpt` receives
// the state gradient behind every run of `run` chunks but the last.
template <typename T, bool kForward, int R>
__global__ void __launch_bounds__(kThreads)
wkv7_chain_kernel(int Tlen, int H, int run, const T* __restrict__ w, const T* __restrict__ r, const T* __restrict__ k,
                  const T* __restrict__ v, const T* __restrict__ a, const T* __restrict__ b, const T* __restrict__ x0,
                  const uint32_t* __restrict__ length, const uint8_t* __restrict__ new_starts, T* __restrict__ y,
                  T* __restrict__ out, float* __restrict__ ckpt, const int* __restrict__ run_if, int run_ticket,
                  int* __restrict__ residual_mark) {
    // Behind the chunked kernels: run only when the forward met something outside their domain (it left its ticket), and
    // backward only when the residual is marked as these kernels'.
    if (run_if != nullptr) {
        const int word = word_behind(run_if);
        if (kForward ? word != run_ticket : word == 0) return;
    }
    if (kForward && residual_mark != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *residual_mark = 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ChainSmem<R>& sm = *reinterpret_cast<ChainSmem<R>*>(smem_raw);
    constexpr int kRows = 8 * R, kParts = kN / kRows;
    const int bh = blockIdx.x / kParts, part = blockIdx.x % kParts, bi = bh / H, h = bh % H;
    const int tid = threadIdx.x;
    const bool streamer = tid >= kCompute;
    const size_t seq_base = (size_t)bi * Tlen * H * kN + (size_t)h * kN;
    const size_t tok_stride = (size_t)H * kN;
    const uint8_t* ns = new_starts + (size_t)bi * Tlen;
    const int L = min((int)length[bi], Tlen);
    const int nC = (Tlen + kExactChunk - 1) / kExactChunk;

    auto chunk = [&](int ci) { return kForward ? ci : nC - 1 - ci; };      // walking order

    // ---- streaming warps: 16 threads to a token, four channels each; two passes cover a chunk.  A chunk's rows are
    // fetched into registers three chunks ahead (rows behind the end: the last one again), all loads before the first use,
    // and put down in shared memory one chunk ahead: two sets of registers in turn, so that a fetch has more than the time of
    // a whole chunk (about a microsecond) to arrive.
    struct Raw {
        float4 w[2], a[2], b[2], k[2], r[2], rows[2];
        bool start;
    };
    const int q = tid - kCompute, lc = (q & 15) * 4;
    auto fetch = [&](Raw& raw, int ci) {
        if (ci >= nC) return;
        const int c = chunk(ci);
#pragma unroll
        for (int pass = 0; pass < 2; ++pass) {
            const size_t at = seq_base + (size_t)min(c * kExactChunk + (q >> 4) + 8 * pass, Tlen - 1) * tok_stride + lc;
            raw.w[pass] = load4(w + at);
            raw.a[pass] = load4(a + at);
            raw.b[pass] = load4(b + at);
            raw.r[pass] = load4(r + at);
            if (kForward) raw.k[pass] = load4(k + at);
            if ((q & 15) < kRows / 4 && v != nullptr) raw.rows[pass] = load4(v + at + part * kRows);   // the CTA's own rows of v or dy
        }
        raw.start = q < kExactChunk && ns[min(c * kExactChunk + q, Tlen - 1)] != 0;
    };
    auto put = [&](const Raw& raw, int ci) {
        if (ci >= nC) return;
        const int c = chunk(ci), buf = ci & 1;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int pass = 0; pass < 2; ++pass) {
            const int i = (q >> 4) + 8 * pass;
            const bool in = c * kExactChunk + i < Tlen;
            // tokens behind the end leave x as it is
            *reinterpret_cast<float4*>(&sm.vec[buf][kW][i][lc]) = in ? decay4(raw.w[pass]) : make_float4(1.f, 1.f, 1.f, 1.f);
            *reinterpret_cast<float4*>(&sm.vec[buf][kA][i][lc]) = in ? raw.a[pass] : zero;
            *reinterpret_cast<float4*>(&sm.vec[buf][kB][i][lc]) = in ? raw.b[pass] : zero;
            *reinterpret_cast<float4*>(&sm.vec[buf][kR][i][lc]) = in ? raw.r[pass] : zero;
            if (kForward) *reinterpret_cast<float4*>(&sm.vec[buf][kK][i][lc]) = in ? raw.k[pass] : zero;
            if ((q & 15) < kRows / 4) *reinterpret_cast<float4*>(&sm.rows[buf][i][lc]) = in && v != nullptr ? raw.rows[pass] : zero;
        }
        if (q < 32) {
            const uint32_t f = __ballot_sync(0xffffffffu, raw.start && c * kExactChunk + q < Tlen);
            if (q == 0) sm.starts[buf] = f;
        }
    };
    auto flush_y = [&](int c) {
        constexpr int kQuads = kRows / 4;
        const int buf = c & 1, i = q / kQuads, cc = (q % kQuads) * 4, t = c * kExactChunk + i;
        if (q < kQuads * kExactChunk && t < Tlen)
            store4(y + seq_base + (size_t)t * tok_stride + part * kRows + cc, *reinterpret_cast<const float4*>(&sm.y[buf][i][cc]));
    };

    // ---- computing warps
    const int p = tid & 7, row = ((tid >> 3) * R) & (kRows - 1);             // rows `row` .. row + R - 1
    const size_t row_at = ((size_t)bh * kN + part * kRows + row) * kN;
    Cols x[R];
    auto clear = [&]() {
#pragma unroll
        for (int n = 0; n < R; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) x[n].v[e].u = 0;
    };
    auto store_rows = [&](auto* to) {
#pragma unroll
        for (int n = 0; n < R; ++n) store_cols(to + n * kN, p, x[n]);
    };
    auto add_rows = [&](const T* from) {
#pragma unroll
        for (int m = 0; m < R; ++m) {
            const Cols g = load_cols(from + m * kN, p);
#pragma unroll
            for (int e = 0; e < 4; ++e) x[m].v[e] = add2(x[m].v[e], g.v[e]);
        }
    };
    clear();
    if (kForward && !streamer) {
#pragma unroll
        for (int n = 0; n < R; ++n) x[n] = load_cols(x0 + row_at + n * kN, p);
        if (L == 0) store_rows(out + row_at);
    }
    if (streamer) {
        Raw even, odd;
        fetch(even, 0);
        put(even, 0);
        fetch(odd, 1);
        fetch(even, 2);
        __syncthreads();
        for (int ci = 0; ci < nC; ci += 2) {
            if (kForward && ci > 0) flush_y(ci - 1);
            put(odd, ci + 1);
            fetch(odd, ci + 3);
            __syncthreads();
            if (ci + 1 == nC) break;
            if (kForward) flush_y(ci);
            put(even, ci + 2);
            fetch(even, ci + 4);
            __syncthreads();
        }
        if (kForward) flush_y(nC - 1);
        return;
    }
    __syncthreads();
    for (int ci = 0; ci < nC; ++ci) {
        const int c = chunk(ci), buf = ci & 1, t0 = c * kExactChunk;
        const uint32_t starts = sm.starts[buf];
        const size_t in_ckpt = (size_t)(part * kRows + row) * kN;
        if (kForward) {
            if (ckpt != nullptr) store_rows(ckpt + ((size_t)bh * nC + c) * kN * kN + in_ckpt);
        } else if (c + 1 < nC && (c + 1) % run == 0) {
            store_rows(ckpt + ((size_t)bh * ((nC - 1) / run) + c / run) * kN * kN + in_ckpt);
        }
        // Nearly every chunk has neither a start flag nor the returned state inside: its steps are free of branches, so
        // that a token's shared-memory reads are under way while the one before it waits for its sum.
        struct Vecs { Cols W, A, U, K, Y; float v[R]; };   // a token's vectors: forward w, a, b, k, r; backward w, b, a, r
        auto vecs = [&](int i) {
            Vecs m;
            m.W = cols(sm.vec[buf][kW][i], p);
            m.A = cols(sm.vec[buf][kForward ? kA : kB][i], p);
            m.U = cols(sm.vec[buf][kForward ? kB : kA][i], p);
            m.K = cols(sm.vec[buf][kForward ? kK : kR][i], p);
            if (kForward) m.Y = cols(sm.vec[buf][kR][i], p);
#pragma unroll
            for (int n = 0; n < R; ++n) m.v[n] = sm.rows[buf][i][row + n];
            return m;
        };
        auto index = [&](int i) { return kForward ? i : kExactChunk - 1 - i; };
        constexpr int kGroup = 8 / R;             // tokens whose R outputs each are summed over the eight lanes together
        auto walk = [&](auto plain) {
            Vecs next = vecs(index(0));
#pragma unroll 1
            for (int group = 0; group < kExactChunk; group += kGroup) {
                float yp[8];
#pragma unroll
                for (int j = 0; j < kGroup; ++j) {
                    const int i = index(group + j);
                    const Vecs m = next;
                    next = vecs(index((group + j + 1) % kExactChunk));    // a token ahead: under way while this one waits for its sums
                    if (kForward) {
                        if (!plain.value && ((starts >> i) & 1u)) clear();
                        float s[R];
#pragma unroll
                        for (int n = 0; n < R; ++n) s[n] = sum8(dot(x[n], m.A));
#pragma unroll
                        for (int n = 0; n < R; ++n) {
                            const Pair S = pair(s[n], s[n]), V = pair(m.v[n], m.v[n]);
#pragma unroll
                            for (int e = 0; e < 4; ++e) x[n].v[e] = fma2(S, m.U.v[e], fma2(x[n].v[e], m.W.v[e], mul2(V, m.K.v[e])));
                            yp[R * j + n] = dot(x[n], m.Y);
                        }
                        if (!plain.value && t0 + i == L - 1) store_rows(out + row_at);
                    } else {
                        if (!plain.value && t0 + i == L - 1 && x0 != nullptr) add_rows(x0 + row_at);
                        float s[R];
#pragma unroll
                        for (int n = 0; n < R; ++n) {
                            const Pair V = pair(m.v[n], m.v[n]);
#pragma unroll
                            for (int e = 0; e < 4; ++e) x[n].v[e] = fma2(V, m.K.v[e], x[n].v[e]);
                            s[n] = sum8(dot(x[n], m.A));
                        }
#pragma unroll
                        for (int n = 0; n < R; ++n) {
                            const Pair S = pair(s[n], s[n]);
#pragma unroll
                            for (int e = 0; e < 4; ++e) x[n].v[e] = fma2(S, m.U.v[e], mul2(x[n].v[e], m.W.v[e]));
                        }
                        if (!plain.value && ((starts >> i) & 1u)) clear();
                    }
                }
                if (kForward) {
                    const float sum = transpose_sum8(yp, p);     // of token group + p / R, row p % R
                    sm.y[buf][group + p / R][row + p % R] = sum;
                }
            }
        };
        if (starts == 0 && (L <= t0 || L > t0 + kExactChunk)) walk(Plain()); else walk(Marked());
        __syncthreads();
    }
    if (!kForward) {
        if (L == 0 && x0 != nullptr) add_rows(x0 + row_at);
        store_rows(out + row_at);
    }
}

template <typename T, bool kForward, int R>
int launch_rows(cudaStream_t st, int B, int Tlen, int H, int run, const void* w, const void* r, const void* k, const void* v,
                const void* a, const void* b, const void* x0, const uint32_t* length, const uint8_t* ns, void* y, void* out,
                float* ckpt, const int* run_if, int run_ticket, int* residual_mark) {
    auto kern = wkv7_chain_kernel<T, kForward, R>;
    const int smem = (int)sizeof(ChainSmem<R>);
    static DeviceOnce smem_attr;   // one per template instance; the attribute is per device
    if (!smem_attr.ok([kern, smem]() { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); }))
        return B200WKV_ELAUNCH;
    if (run_if != nullptr)
        return launch_behind(kern, B * H * (8 / R), kThreads, smem, st, Tlen, H, run, (const T*)w, (const T*)r, (const T*)k, (const T*)v, (const T*)a,
                             (const T*)b, (const T*)x0, length, ns, (T*)y, (T*)out, ckpt, run_if, run_ticket, residual_mark) == cudaSuccess
                   ? B200WKV_OK
                   : B200WKV_ELAUNCH;
    kern<<<B * H * (8 / R), kThreads, smem, st>>>(Tlen, H, run, (const T*)w, (const T*)r, (const T*)k, (const T*)v, (const T*)a, (const T*)b,
                                                  (const T*)x0, length, ns, (T*)y, (T*)out, ckpt, run_if, run_ticket, residual_mark);
    return cudaGetLastError() == cudaSuccess ? B200WKV_OK : B200WKV_ELAUNCH;
}
// Few rows per lane while the CTAs find SMs of their own, more when they have to share them.  Measured (fp32, us for forward
// + backward chain; R = 1, 2, 4): 8 heads, T = 256: 62, 76, 102; 48 heads, T = 256: 153, 92, 104; 128 heads, T = 256: 312,
// 186, 123; 640 heads, T = 200: 1129, 671, 485.
int rows_per_lane(int heads) {
    const int sms = sm_count_of_current_device();
    return 8 * heads <= sms ? 1 : 2 * heads <= sms ? 2 : 4;
}
template <typename T, bool kForward, typename... Args>
int launch_chain(cudaStream_t st, int B, int Tlen, int H, Args... args) {
    switch (rows_per_lane(B * H)) {
        case 1: return launch_rows<T, kForward, 1>(st, B, Tlen, H, args...);
        case 2: return launch_rows<T, kForward, 2>(st, B, Tlen, H, args...);
        default: return launch_rows<T, kForward, 4>(st, B, Tlen, H, args...);
    }
}
}  // namespace

int wkv7_seq_fwd(cudaStream_t st, int dtype, int B, int T, int H, const void* w, const void* r, const void* k, const void* v,
                 const void* a, const void* b, const void* s0, const uint32_t* length, const uint8_t* ns, void* y, void* s_out,
                 void* residual, const int* run_if, int run_ticket, int* residual_mark) {
    auto launch = [&](auto type) {
        return launch_chain<decltype(type), true>(st, B, T, H, 0, w, r, k, v, a, b, s0, length, ns, y, s_out, (float*)residual, run_if,
                                                  run_ticket, residual_mark);
    };
    return dtype == B200WKV_F32 ? launch(float()) : launch(__nv_bfloat16());
}
int wkv7_chain_bwd(cudaStream_t st, int dtype, int B, int T, int H, int run, const void* w, const void* r, const void* a, const void* b,
                   const void* dy, const void* ds_out, const uint32_t* length, const uint8_t* ns, void* ds0, float* carry, const int* run_if) {
    auto launch = [&](auto type) {
        return launch_chain<decltype(type), false>(st, B, T, H, run, w, r, (const void*)nullptr, dy, a, b, ds_out, length, ns, (void*)nullptr, ds0,
                                                   carry, run_if, 0, (int*)nullptr);
    };
    return dtype == B200WKV_F32 ? launch(float()) : launch(__nv_bfloat16());
}

}  // namespace b200wkv
