// RWKV-4 WKV recurrence as a scan over time segments, fp32 arithmetic.
//
// Per channel the state is (aa, bb, pp): numerator, denominator and the exponent both are scaled
// by.  With w' = -exp(w) (jaxrwkv src/jaxrwkv/rwkv4.py:312) and u = time_first:
//   q  = max(pp, u + k_t)      y_t = (e^{pp-q} aa + e^{u+k_t-q} v_t) / (e^{pp-q} bb + e^{u+k_t-q})
//   q' = max(pp + w', k_t)     aa <- e^{pp+w'-q'} aa + e^{k_t-q'} v_t,  bb likewise with 1,  pp <- q'
// A start flag resets the state to (0, 0, -1e30).  Semantics: BaseRWKV.inner_loop, rwkv4.py:143-172.
//
// One thread per (sequence, channel) walking all T tokens is bound by the token-to-token latency (0.35 us per token
// forward, 0.95 us backward: 1.3 ms for T = 1024 however few channels there are).  The recurrence is associative, so
// here a CTA of eight warps owns 32 channels of one sequence, each warp consecutive segments of 16 tokens, and up to four
// CTAs of a cluster own consecutive runs of 128 tokens:
//   1. every warp reduces its segment to a summary, starting from the empty state;
//   2. the summaries are combined in order, inside the CTA and then across the cluster through distributed shared
//      memory (each thread for its channel; the exponents form a short max-plus chain, the exponentials hang off it in
//      parallel), which gives every segment its entering state;
//   3. every warp walks its segment again from that state and writes the results.
// The cluster then moves on by its 512 tokens with the combined state as carry.  Of the two exponentials of an update
// one is always 1, so an update costs one.
//
// Backward: the state entering every segment is a checkpoint of the forward.  y depends on the state only through
// A = aa e^pp and B = bb e^pp, so the cotangent of pp is aa gaa + bb gbb plus a part z that only the cotangent of the
// RETURNED state can have and that follows the arguments of the running maximum back:
//   gaa' = e1 gaa + (output term),  gbb' likewise,  z' = z while the maximum is the old exponent, else z goes to k_t.
// That is linear in (gaa, gbb, z) with a scalar factor per segment, so the same three steps apply, in reverse order of
// segments; step 1 can be computed walking FORWARD with the running product of the factors, together with the replay
// of the states.  What the replay computed (states, weights, reciprocals) stays in registers for step 3.
// 1340 us -> 48 us forward + 94 us backward at B=8, T=1024, C=768, bf16 (75 and 102 MB of streams; under ncu, cold).  No unit is
// full: issue slots 59 and 47 %, DRAM 10 %, 21 and 15 warps per SM (80 and 128 registers).  Per issued instruction a warp waits
// 2.1 and 1.4 cycles for its rows out of global memory, which all come at a segment's start, and 1.0 and 0.8 for the cluster's
// fences.
#include <cooperative_groups.h>
#include "common.cuh"
#include "device_once.cuh"
#include "host_calls.h"

namespace b200wkv {

namespace {
constexpr int kSeg = 16;        // tokens per segment = per checkpoint
constexpr float kEmpty = -1e30f;

constexpr int kWarps = 8;       // segments of a CTA
constexpr int kMaxCluster = 4;  // CTAs of a cluster
namespace cg = cooperative_groups;

// e^{-|d|}.  The weights it makes are at most 1 and the other weight of the same sum is 1: an error of |d| 2^-24 e^{-|d|}
// stays below the rounding of the sum.
__device__ __forceinline__ float exp_neg_abs(float d) {
    float e;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(fabsf(d) * -1.4426950408889634f));
    return e;
}
// weights of the old (e1) and the new (e2) part under the common exponent max(x, y); returns whether x is the maximum
__device__ __forceinline__ bool split_weights(float x, float y, float& e1, float& e2) {
    const float d = x - y;
    const float e = exp_neg_abs(d);
    const bool first = d >= 0.f;
    e1 = first ? 1.f : e;
    e2 = first ? e : 1.f;
    return first;
}

// 1 / x to the last bit or two without the branch of the IEEE division's special cases (which would cut the instruction
// stream at every token): the hardware's approximation and one Newton step; 0 and infinities keep its answer.
__device__ __forceinline__ float reciprocal(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    const float e = fmaf(-x, r, 1.f);
    return fabsf(e) < 0.5f ? fmaf(r, e, r) : r;
}

// Two streams' values of one token in as few registers as they take (one for bf16): the raw rows of a segment stay in
// registers from the first walk to the second.
template <typename T> struct Two;
template <> struct Two<float> {
    float a, b;
    __device__ __forceinline__ void set(float x, float y) { a = x; b = y; }
    __device__ __forceinline__ float x() const { return a; }
    __device__ __forceinline__ float y() const { return b; }
};
template <> struct Two<__nv_bfloat16> {
    uint32_t raw;
    __device__ __forceinline__ void set(__nv_bfloat16 x, __nv_bfloat16 y) {
        raw = (uint32_t)__bfloat16_as_ushort(x) | ((uint32_t)__bfloat16_as_ushort(y) << 16);
    }
    __device__ __forceinline__ float x() const { return __uint_as_float(raw << 16); }
    __device__ __forceinline__ float y() const { return __uint_as_float(raw & 0xffff0000u); }
};
// A segment of kSeg tokens in which the returned state is not taken has no branch in its walks: all its loads are in
// flight at once and the tokens' exponentials overlap.  The other kind: the sequence's last segment, and `length`'s.
struct Full { static constexpr bool value = true; };
struct Ragged { static constexpr bool value = false; };

// The exponential that split_weights computes, carrying which of the two weights it is as its sign bit: negative when the
// second is 1 and the exponential belongs to the first.
__device__ __forceinline__ float signed_weight(float x, float y) {
    const float d = x - y;
    return copysignf(exp_neg_abs(d), d >= 0.f ? 1.f : -1.f);
}
__device__ __forceinline__ bool from_signed(float s, float& e1, float& e2) {
    const bool first = !signbit(s);
    const float e = fabsf(s);
    e1 = first ? 1.f : e;
    e2 = first ? e : 1.f;
    return first;
}

// start flags of the segment that begins at t0 as a bit mask (bit i = token t0 + i)
__device__ __forceinline__ uint32_t segment_flags(const uint8_t* ns, int t0, int Tlen, int lane) {
    const bool f = lane < kSeg && t0 + lane < Tlen && ns[t0 + lane] != 0;
    return __ballot_sync(0xffffffffu, f);
}

// the decay -exp(w), rounded to the element type as the reference stores it; `raw` = the caller has not applied it
template <typename T>
__device__ __forceinline__ float decay_of(T w, bool raw) {
    return raw ? to_f32(from_f32<T>(-expf(to_f32(w)))) : to_f32(w);
}

// The log-decay over n tokens: 0 over none, also where one token's is infinite (exp(w) out of range).
__device__ __forceinline__ float decay_over(int n, float ww) { return n > 0 ? (float)n * ww : 0.f; }
// State (a, b, p) followed by a stretch of tokens with summary (xa, xb, xp) that decays it by `decay` or, with `cut`, drops it
// (whatever it is: a NaN in front of a start flag ends there).
__device__ __forceinline__ void combine(float& a, float& b, float& p, bool cut, float decay, float xa, float xb, float xp) {
    float e1, e2;
    const float x = p + decay;
    split_weights(x, xp, e1, e2);
    a = cut ? xa : e1 * a + e2 * xa; b = cut ? xb : e1 * b + e2 * xb; p = cut ? xp : fmaxf(x, xp);
}
// factor x, with nothing left of x where the factor is 0: a start flag lies between
__device__ __forceinline__ float carried(float factor, float x) { return factor != 0.f ? factor * x : 0.f; }

template <typename T>
__global__ void __launch_bounds__(kWarps * 32, 3)
wkv4_fwd_kernel(int Tlen, int C, bool raw_w, const T* __restrict__ w, const T* __restrict__ u, const T* __restrict__ r,
                const T* __restrict__ k, const T* __restrict__ v, const T* __restrict__ s0,
                const uint32_t* __restrict__ length, const uint8_t* __restrict__ new_starts, T* __restrict__ s_out,
                T* __restrict__ y, float* __restrict__ ckpt) {
    __shared__ float sa[kWarps][32], sb[kWarps][32], sp[kWarps][32];
    __shared__ float cta_sum[3][32];        // the whole CTA's summary, read by the other CTAs of the cluster
    __shared__ int sreset[kWarps], cta_reset;
    const cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int groups = (C + 31) / 32, unit = blockIdx.x / ranks, bi = unit / groups, c = (unit % groups) * 32 + lane;
    const bool live = c < C;
    const int cc = live ? c : C - 1;
    const int L = min((int)length[bi], Tlen);
    const int nC = (Tlen + kSeg - 1) / kSeg;
    const float ww = decay_of<T>(w[cc], raw_w), uu = to_f32(u[cc]);
    const size_t so = (size_t)bi * 3 * C + cc;
    float ca = to_f32(s0[so]), cb = to_f32(s0[so + C]), cp = to_f32(s0[so + 2 * C]);   // state entering the segments at hand
    if (L == 0 && warp == 0 && rank == 0 && live) { s_out[so] = s0[so]; s_out[so + C] = s0[so + C]; s_out[so + 2 * C] = s0[so + 2 * C]; }
    const size_t base = (size_t)bi * Tlen * C + cc;
    const uint8_t* ns = new_starts + (size_t)bi * Tlen;
    for (int g00 = 0; g00 < nC; g00 += kWarps * ranks) {
        const int g0 = g00 + rank * kWarps, seg = g0 + warp, t0 = seg * kSeg, n = min(kSeg, Tlen - t0);   // n <= 0: nothing of the sequence is left
        const bool full_seg = n == kSeg && (L <= t0 || L >= t0 + kSeg);
        const bool ends = full_seg && L == t0 + kSeg;      // the returned state is the one behind this segment
        Two<T> kv[kSeg];
        if (n > 0) {
#pragma unroll
            for (int i = 0; i < kSeg; ++i) {   // rows behind the end: the last one again, unused
                const size_t at = base + (size_t)(t0 + min(i, n - 1)) * C;
                kv[i].set(k[at], v[at]);
            }
        }
        const uint32_t starts = segment_flags(ns, t0, Tlen, lane);
        // 1. summary
        float a = 0.f, b = 0.f, p = kEmpty;
        auto summarise = [&](auto full) {
#pragma unroll
            for (int i = 0; i < kSeg; ++i)
                if (full.value || i < n) {
                    const bool start = (starts >> i) & 1u;
                    a = start ? 0.f : a; b = start ? 0.f : b; p = start ? kEmpty : p;
                    float e1, e2;
                    const float x = p + ww, kt = kv[i].x();
                    split_weights(x, kt, e1, e2);
                    a = e1 * a + e2 * kv[i].y(); b = e1 * b + e2; p = fmaxf(x, kt);
                }
        };
        if (full_seg) summarise(Full()); else summarise(Ragged());
        sa[warp][lane] = a; sb[warp][lane] = b; sp[warp][lane] = p;
        if (lane == 0) sreset[warp] = starts != 0;
        __syncthreads();
        // 2. the CTA's own summary up to each of its segments (a, b, p with `cut` = a start flag inside), then the carry
        //    brought forward through the CTAs in front, to this CTA and to the end of the cluster
        float xa = 0.f, xb = 0.f, xp = kEmpty;      // summary of the CTA's segments so far
        bool cut = false, own_cut = false;
        int own_n = 0, cta_n = 0;
        a = 0.f; b = 0.f; p = kEmpty;
#pragma unroll
        for (int j = 0; j < kWarps; ++j) {
            if (j == warp) { a = xa; b = xb; p = xp; own_cut = cut; own_n = cta_n; }
            const int nj = max(0, min(kSeg, Tlen - (g0 + j) * kSeg));
            const bool rj = sreset[j] != 0;
            combine(xa, xb, xp, rj, decay_over(nj, ww), sa[j][lane], sb[j][lane], sp[j][lane]);
            cut |= rj;
            cta_n += nj;
        }
        if (ranks > 1) {
            if (warp == 0) { cta_sum[0][lane] = xa; cta_sum[1][lane] = xb; cta_sum[2][lane] = xp; }
            if (threadIdx.x == 0) cta_reset = cut;
            cluster.sync();
        }
        float ea = 0.f, eb = 0.f, ep = 0.f;         // state entering this CTA's segments
        for (int q = 0; q < ranks; ++q) {
            if (q == rank) { ea = ca; eb = cb; ep = cp; }
            float qa = xa, qb = xb, qp = xp;
            bool qr = cut;
            if (q != rank) {
                const float* from = cluster.map_shared_rank(&cta_sum[0][0], q);
                qa = from[lane]; qb = from[32 + lane]; qp = from[64 + lane];
                qr = *cluster.map_shared_rank(&cta_reset, q) != 0;
            }
            const int nq = max(0, min(kWarps * kSeg, Tlen - (g00 + q * kWarps) * kSeg));
            combine(ca, cb, cp, qr, decay_over(nq, ww), qa, qb, qp);
        }
        {
            const float xa2 = a, xb2 = b, xp2 = p;
            a = ea; b = eb; p = ep;
            combine(a, b, p, own_cut, decay_over(own_n, ww), xa2, xb2, xp2);
        }
        // 3. outputs
        if (n > 0 && ckpt != nullptr && live) {
            float* q = ckpt + (((size_t)bi * nC + seg) * 3) * C + c;
            q[0] = a; q[C] = b; q[2 * C] = p;
        }
        auto outputs = [&](auto full) {
            T rr[kSeg];
            if (r != nullptr) {
#pragma unroll
                for (int i = 0; i < kSeg; ++i) rr[i] = r[base + (size_t)(t0 + min(i, n - 1)) * C];
            }
#pragma unroll
            for (int i = 0; i < kSeg; ++i)
                if (full.value || i < n) {
                    const bool start = (starts >> i) & 1u;
                    a = start ? 0.f : a; b = start ? 0.f : b; p = start ? kEmpty : p;
                    float e1, e2;
                    const float kt = kv[i].x(), vt = kv[i].y();
                    split_weights(p, uu + kt, e1, e2);
                    float o = (e1 * a + e2 * vt) * reciprocal(e1 * b + e2);
                    if (r != nullptr) o = to_f32(from_f32<T>(o)) * to_f32(rr[i]);   // rounded as where the caller multiplies
                    if (live) y[base + (size_t)(t0 + i) * C] = from_f32<T>(o);
                    const float x = p + ww;
                    split_weights(x, kt, e1, e2);
                    a = e1 * a + e2 * vt; b = e1 * b + e2; p = fmaxf(x, kt);
                    if (!full.value && t0 + i == L - 1 && live) { s_out[so] = from_f32<T>(a); s_out[so + C] = from_f32<T>(b); s_out[so + 2 * C] = from_f32<T>(p); }
                }
        };
        if (full_seg) outputs(Full()); else if (n > 0) outputs(Ragged());
        if (ends && live) { s_out[so] = from_f32<T>(a); s_out[so + C] = from_f32<T>(b); s_out[so + 2 * C] = from_f32<T>(p); }
        if (ranks > 1) cluster.sync(); else __syncthreads();   // the summaries are read before the next ones are written
    }
}

template <typename T>
__global__ void __launch_bounds__(kWarps * 32, sizeof(T) == 2 ? 2 : 1)
wkv4_bwd_kernel(int Tlen, int C, bool raw_w, const T* __restrict__ w, const T* __restrict__ u, const T* __restrict__ r,
                const T* __restrict__ k, const T* __restrict__ v, const T* __restrict__ gy,
                const uint32_t* __restrict__ length, const uint8_t* __restrict__ new_starts, const T* __restrict__ gs_new,
                const float* __restrict__ ckpt, float* __restrict__ gw, float* __restrict__ gu, T* __restrict__ gr,
                T* __restrict__ gk, T* __restrict__ gv, T* __restrict__ gs) {
    // per segment: cotangents (numerator, denominator, z) of its entering state from inside the segment, the factor of
    // the first two and (as 0 or 1) of z
    __shared__ float sa[kWarps][32], sb[kWarps][32], sz[kWarps][32], se[kWarps][32], sf[kWarps][32];
    __shared__ float cta_sum[5][32];            // the same of the whole CTA, read by the other CTAs of the cluster
    const cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int groups = (C + 31) / 32, unit = blockIdx.x / ranks, bi = unit / groups, c = (unit % groups) * 32 + lane;
    const bool live = c < C;
    const int cc = live ? c : C - 1;
    const int L = min((int)length[bi], Tlen);
    const int nC = (Tlen + kSeg - 1) / kSeg;
    const float ww = decay_of<T>(w[cc], raw_w), uu = to_f32(u[cc]);
    const size_t so = (size_t)bi * 3 * C + cc, base = (size_t)bi * Tlen * C + cc;
    const uint8_t* ns = new_starts + (size_t)bi * Tlen;
    float gsa = 0.f, gsb = 0.f, gsp = 0.f;
    if (gs_new != nullptr) { gsa = to_f32(gs_new[so]); gsb = to_f32(gs_new[so + C]); gsp = to_f32(gs_new[so + 2 * C]); }
    float ca = 0.f, cb = 0.f, cz = 0.f;       // cotangent of the state behind the segments at hand
    float gw_acc = 0.f, gu_acc = 0.f;
    const int step = kWarps * ranks;
    for (int g00 = (nC - 1) / step * step; g00 >= 0; g00 -= step) {
        const int g0 = g00 + rank * kWarps, seg = g0 + warp, t0 = seg * kSeg, n = min(kSeg, Tlen - t0);
        const bool full_seg = n == kSeg && (L <= t0 || L >= t0 + kSeg);
        const bool ends = full_seg && L == t0 + kSeg;      // the returned state is the one behind this segment
        const uint32_t starts = segment_flags(ns, t0, Tlen, lane);
        // what the replay leaves for the way back: state entering each token (after a reset), the reciprocal of y's
        // denominator, and the exponential of the update and of the output with the sign that says which weight it is
        float ha[kSeg], hb[kSeg], hinv[kSeg], hs[kSeg], ho[kSeg];
        float a = 0.f, b = 0.f, p = kEmpty, a_in = 0.f, b_in = 0.f;
        if (n > 0) {
            const float* q = ckpt + (((size_t)bi * nC + seg) * 3) * C + cc;
            a = q[0]; b = q[C]; p = q[2 * C];
        }
        a_in = a; b_in = b;
        // 1. replay of the states and, in the same walk, what the segment adds to the cotangent of its entering state:
        //    each token's term times the product of the factors in front of it
        float xa = 0.f, xb = 0.f, xz = 0.f, pe = 1.f, pf = 1.f;
        Two<T> kv[kSeg], gr_[kSeg];           // k, v and the cotangent, the receptance of every token
        auto replay = [&](auto full) {
#pragma unroll
            for (int i = 0; i < kSeg; ++i) {   // rows behind the end: the last one again, unused
                    const size_t at = base + (size_t)(t0 + min(i, n - 1)) * C;
                    kv[i].set(k[at], v[at]);
                    gr_[i].set(gy != nullptr ? gy[at] : from_f32<T>(0.f), r != nullptr ? r[at] : from_f32<T>(1.f));
                }
#pragma unroll
            for (int i = 0; i < kSeg; ++i)
                if (full.value || i < n) {
                    const bool start = (starts >> i) & 1u;
                    a = start ? 0.f : a; b = start ? 0.f : b; p = start ? kEmpty : p;
                    pe = start ? 0.f : pe; pf = start ? 0.f : pf;
                    ha[i] = a; hb[i] = b;
                    const float kt = kv[i].x(), vt = kv[i].y();
                    float e1, e2;
                    ho[i] = signed_weight(p, uu + kt);
                    from_signed(ho[i], e1, e2);
                    const float num = e1 * a + e2 * vt, inv = reciprocal(e1 * b + e2);
                    hinv[i] = inv;
                    const float gnum = gr_[i].x() * gr_[i].y() * inv, gden = -gnum * num * inv;
                    xa += carried(pe, e1 * gnum); xb += carried(pe, e1 * gden);
                    const float x = p + ww;
                    hs[i] = signed_weight(x, kt);
                    const bool first = from_signed(hs[i], e1, e2);
                    a = e1 * a + e2 * vt; b = e1 * b + e2; p = fmaxf(x, kt);
                    pe = carried(pe, e1);
                    if (!first) pf = 0.f;
                    if (!full.value && t0 + i == L - 1) {    // the returned state's cotangent enters behind token L - 1
                        xa += carried(pe, gsa); xb += carried(pe, gsb);
                        xz += carried(pf, gsp - a * gsa - b * gsb);
                    }
                }
        };
        if (full_seg) replay(Full()); else if (n > 0) replay(Ragged());
        if (ends) {
            xa += carried(pe, gsa); xb += carried(pe, gsb);
            xz += carried(pf, gsp - a * gsa - b * gsb);
        }
        sa[warp][lane] = xa; sb[warp][lane] = xb; sz[warp][lane] = xz; se[warp][lane] = pe; sf[warp][lane] = pf;
        __syncthreads();
        // 2. the CTA's own sums behind each of its segments, then the carry brought back through the CTAs behind, to
        //    this CTA and to the start of the cluster
        float qe = 1.f, qf = 1.f, qa = 0.f, qb = 0.f, qz = 0.f, own_e = 1.f, own_f = 1.f, ga = 0.f, gb = 0.f, z = 0.f;
#pragma unroll
        for (int j = kWarps - 1; j >= 0; --j) {
            if (j == warp) { own_e = qe; own_f = qf; ga = qa; gb = qb; z = qz; }
            const float ej = se[j][lane], fj = sf[j][lane];
            qa = carried(ej, qa) + sa[j][lane]; qb = carried(ej, qb) + sb[j][lane]; qz = carried(fj, qz) + sz[j][lane];
            qe = qe != 0.f ? carried(ej, qe) : 0.f; qf *= fj;
        }
        if (ranks > 1) {
            if (warp == 0) { cta_sum[0][lane] = qa; cta_sum[1][lane] = qb; cta_sum[2][lane] = qz; cta_sum[3][lane] = qe; cta_sum[4][lane] = qf; }
            cluster.sync();
        }
        float ia = 0.f, ib = 0.f, iz = 0.f;         // cotangent behind this CTA's segments
        for (int q = ranks - 1; q >= 0; --q) {
            float ra = qa, rb = qb, rz = qz, re = qe, rf = qf;
            if (q == rank) { ia = ca; ib = cb; iz = cz; }
            else {
                const float* from = cluster.map_shared_rank(&cta_sum[0][0], q) + lane;
                ra = from[0]; rb = from[32]; rz = from[64]; re = from[96]; rf = from[128];
            }
            ca = carried(re, ca) + ra; cb = carried(re, cb) + rb; cz = carried(rf, cz) + rz;
        }
        ga += carried(own_e, ia); gb += carried(own_e, ib); z += carried(own_f, iz);
        // 3. gradients, walking back through the segment
        if (ends) { ga += gsa; gb += gsb; z += gsp - a * gsa - b * gsb; }   // (a, b): the state behind the segment
        auto gradients = [&](auto full) {
#pragma unroll
            for (int i = kSeg - 1; i >= 0; --i)
                if (full.value || i < n) {
                    const size_t at = base + (size_t)(t0 + i) * C;
                    const float vt = kv[i].y(), go = gr_[i].x();
                    const float a0 = ha[i], b0 = hb[i], inv = hinv[i];
                    float e1, e2;
                    const bool first = from_signed(hs[i], e1, e2);
                    if (!full.value && t0 + i == L - 1) {
                        ga += gsa; gb += gsb;
                        z += gsp - (e1 * a0 + e2 * vt) * gsa - (e1 * b0 + e2) * gsb;
                    }
                    gw_acc += e1 * (a0 * ga + b0 * gb) + (first ? z : 0.f);
                    float gkt = e2 * (vt * ga + gb) + (first ? 0.f : z);
                    float gvt = e2 * ga;
                    ga *= e1; gb *= e1;
                    if (!first) z = 0.f;
                    from_signed(ho[i], e1, e2);
                    const float o = (e1 * a0 + e2 * vt) * inv;
                    const float gnum = go * gr_[i].y() * inv, gden = -gnum * o;
                    const float gx = e2 * (vt * gnum + gden);
                    gu_acc += gx; gkt += gx; gvt += e2 * gnum;
                    ga += e1 * gnum; gb += e1 * gden;
                    if (live) {
                        gk[at] = from_f32<T>(gkt);
                        gv[at] = from_f32<T>(gvt);
                        if (r != nullptr) gr[at] = from_f32<T>(go * o);
                    }
                    const bool start = (starts >> i) & 1u;
                    ga = start ? 0.f : ga; gb = start ? 0.f : gb; z = start ? 0.f : z;
                }
        };
        if (full_seg) gradients(Full()); else gradients(Ragged());
        if (g0 == 0 && warp == 0) {           // the sequence's first segment
            float gp = a_in * ga + b_in * gb + z;
            if (L == 0) { ga += gsa; gb += gsb; gp += gsp; }
            if (live) { gs[so] = from_f32<T>(ga); gs[so + C] = from_f32<T>(gb); gs[so + 2 * C] = from_f32<T>(gp); }
        }
        if (ranks > 1) cluster.sync(); else __syncthreads();
    }
    // the shares of dw' and du, added in a fixed order: the CTA's warps, then the CTAs
    sa[warp][lane] = gw_acc; sb[warp][lane] = gu_acc;
    __syncthreads();
    gw_acc = 0.f; gu_acc = 0.f;
#pragma unroll
    for (int j = 0; j < kWarps; ++j) { gw_acc += sa[j][lane]; gu_acc += sb[j][lane]; }
    if (ranks > 1) {
        if (warp == 0) { cta_sum[0][lane] = gw_acc; cta_sum[1][lane] = gu_acc; }
        cluster.sync();
        if (rank == 0 && warp == 0)
            for (int q = 1; q < ranks; ++q) {
                const float* from = cluster.map_shared_rank(&cta_sum[0][0], q) + lane;
                gw_acc += from[0]; gu_acc += from[32];
            }
        cluster.sync();                         // no CTA leaves while its sums are being read
    }
    if (rank == 0 && warp == 0 && live) {
        gw[(size_t)bi * C + c] = gw_acc;
        gu[(size_t)bi * C + c] = gu_acc;
    }
}

template <typename T>
__global__ void wkv4_parameter_grads_kernel(int B, int C, const T* __restrict__ w, const float* gw, const float* gu, T* __restrict__ dw, T* __restrict__ du) {
    wait_for_grid_in_front();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    float sw = 0.f, su = 0.f;
    for (int b = 0; b < B; ++b) { sw += gw[(size_t)b * C + c]; su += gu[(size_t)b * C + c]; }
    dw[c] = from_f32<T>(sw * decay_of<T>(w[c], true));   // d(-exp(w))/dw = -exp(w)
    du[c] = from_f32<T>(su);
}

// One CTA per 128 tokens of a sequence, up to four: CTAs of different time runs spread a small B * C over the SMs.  At
// B=8, T=1024, C=768 clusters of 1 / 2 / 4 / 8 took 150 / 154 / 141 / 170 us in all: eight find room for a whole cluster
// too seldom and wait for one another too long.
int cluster_size(int Tlen) {
    int n = 1;
    while (n < kMaxCluster && n * kWarps * kSeg < Tlen) n *= 2;
    return n;
}
template <typename Kernel, typename... Args>
int launch(Kernel kern, cudaStream_t st, int B, int Tlen, int C, Args... args) {
    const int ranks = cluster_size(Tlen);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ranks; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((C + 31) / 32) * B * ranks);
    cfg.blockDim = dim3(kWarps * 32);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, Tlen, C, args...) == cudaSuccess ? B200WKV_OK : B200WKV_ELAUNCH;
}
}  // namespace

size_t wkv4_residual_bytes(int B, int T, int C) { return (size_t)B * ((T + kSeg - 1) / kSeg) * 3 * C * sizeof(float); }

template <typename T>
static int launch_fwd(cudaStream_t st, int B, int Tlen, int C, bool raw_w, const void* w, const void* u, const void* r, const void* k,
                      const void* v, const void* s0, const uint32_t* length, const uint8_t* ns, void* s_out, void* y, void* residual) {
    return launch(wkv4_fwd_kernel<T>, st, B, Tlen, C, raw_w, (const T*)w, (const T*)u, (const T*)r, (const T*)k, (const T*)v, (const T*)s0,
                  length, ns, (T*)s_out, (T*)y, (float*)residual);
}
template <typename T>
static int launch_bwd(cudaStream_t st, int B, int Tlen, int C, bool raw_w, const void* w, const void* u, const void* r, const void* k,
                      const void* v, const void* gy, const uint32_t* length, const uint8_t* ns, const void* gs_new,
                      const void* residual, float* gw, float* gu, void* gr, void* gk, void* gv, void* gs) {
    return launch(wkv4_bwd_kernel<T>, st, B, Tlen, C, raw_w, (const T*)w, (const T*)u, (const T*)r, (const T*)k, (const T*)v, (const T*)gy,
                  length, ns, (const T*)gs_new, (const float*)residual, gw, gu, (T*)gr, (T*)gk, (T*)gv, (T*)gs);
}

int wkv4_fwd(cudaStream_t st, int dtype, int B, int T, int C, bool raw_w, const void* w, const void* u, const void* r, const void* k,
             const void* v, const void* s0, const uint32_t* length, const uint8_t* ns, void* s_out, void* y, void* residual) {
    return (dtype == B200WKV_F32 ? launch_fwd<float> : launch_fwd<__nv_bfloat16>)(st, B, T, C, raw_w, w, u, r, k, v, s0, length, ns, s_out,
                                                                                  y, residual);
}
int wkv4_bwd(cudaStream_t st, int dtype, int B, int T, int C, bool raw_w, const void* w, const void* u, const void* r, const void* k,
             const void* v, const void* gy, const uint32_t* length, const uint8_t* ns, const void* gs_new, const void* residual,
             float* gw, float* gu, void* gr, void* gk, void* gv, void* gs) {
    return (dtype == B200WKV_F32 ? launch_bwd<float> : launch_bwd<__nv_bfloat16>)(st, B, T, C, raw_w, w, u, r, k, v, gy, length, ns, gs_new,
                                                                                  residual, gw, gu, gr, gk, gv, gs);
}
int wkv4_parameter_grads(cudaStream_t st, int dtype, int B, int C, const void* w, const float* gw, const float* gu, void* dw, void* du) {
    auto launch = [&](auto type) {                // directly behind the backward kernel
        typedef decltype(type) T;
        return launch_behind(wkv4_parameter_grads_kernel<T>, (C + 63) / 64, 64, 0, st, B, C, (const T*)w, gw, gu, (T*)dw, (T*)du);
    };
    return (dtype == B200WKV_F32 ? launch(float()) : launch(__nv_bfloat16())) == cudaSuccess ? B200WKV_OK : B200WKV_ELAUNCH;
}

}  // namespace b200wkv
