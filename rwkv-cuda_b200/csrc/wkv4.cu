// RWKV-4 WKV, fp32, forward and backward.
//
// Operator (wkv/run.py:34-63 of the reference project), per batch b and channel c:
//   y_t = (sum_{s<t} e^{(t-1-s)w+k_s} v_s + e^{u+k_t} v_t) / (sum_{s<t} e^{(t-1-s)w+k_s} + e^{u+k_t})
// Running sums are kept divided by e^{o} (o = running maximum exponent) so nothing overflows.  Of each pair exp(x-max),
// exp(y-max) one is exactly 1, so a step costs one exponential per pair.
//
// A token-by-token walk is a chain of about 160 ns per token with one thread per (b, c): B4 T256 C256 (1024 chains) and
// B32 T768 C768 both waited on it.  The recurrence is linear, so time is split: a block owns 32 channels (its lanes) of one
// batch row and walks time in tiles of S segments (its warps) of L = 8 tokens.  Per tile every warp
//   1. scans its segment from an empty state (its tokens stay in registers, they are read from memory once),
//   2. gets its start state from a scan over the S segments: log2(S) shuffle steps on transposed data in shared memory,
//   3. walks its segment again from that state and writes y.
// Two segments after another are (p, q, o): o = max(o1 + L w, o2), p = p1 e^{o1 + L w - o} + p2 e^{o2 - o}, q alike.
// The backward is the same in reverse, with the adjoint G of the running sums as the state; the running sums themselves
// are rebuilt inside a segment from its start state, which the forward pass leaves once per segment:
//   G_{t-1} = e^w G_t + (1, -y_t) gy_t / den_t      gv_t = A_t + e^{k_t} Gp_t     gk_t = A_t (v_t - y_t) + e^{k_t} (Gp_t v_t + Gq_t)
//   A_t = gy_t e^{u+k_t} / den_t    gu = sum_t A_t (v_t - y_t)    dL/dw = sum_t e^w (Gp_t p_{t-1} + Gq_t q_{t-1})
// Forward + backward of a training step, B32 T768 C768 on a B200: 1111 us token by token, 294 us with a running maximum in every token, 223 us with a test per
// token against the end of the sequence, 203 us here; B4 T256 C256: the two
// kernels took 143 us and take 10 + 12 us now, the whole step is 64 us, host side included.
//
// Compiled without fast-math: the fp32 tolerance of this operator (1e-5) needs accurate expf.
#include "common.cuh"

namespace rwkvb200 {

namespace {

constexpr float kNegInf = -1e38f;
constexpr int L = 8;   // tokens of a segment

struct Sum {           // (p, q) e^{o}
    float p, q, o;
};
struct Pair {
    float a, b, m;
};
// returns a = e^{x-m}, b = e^{y-m}, m = max(x,y) with one exponential
__device__ __forceinline__ Pair softpair(float x, float y) {
    const float d = x - y;
    const float e = expf(-fabsf(d));
    return Pair{d >= 0.f ? 1.f : e, d >= 0.f ? e : 1.f, fmaxf(x, y)};
}
// `first` decayed by `dw` and then `second` added
__device__ __forceinline__ Sum after(Sum first, float dw, Sum second) {
    const Pair s = softpair(first.o + dw, second.o);
    return Sum{s.a * first.p + s.b * second.p, s.a * first.q + s.b * second.q, s.m};
}

// Plain weights.  While the exponents of a segment lie within kSpan of each other (and the start state's with them) they are taken
// relative to the largest once, e_i = e^{k_i - M}, and the recurrences inside the segment are multiply-adds with the constant
// e^w: one exponential per token instead of three forward and six backward.  What such a weight loses by underflow (below
// e^{-87}) is less than 1e-11 of any term that it is added to, because every token's own weight is at least e^{-kSpan - kBonus}.
// A warp with a lane outside the bounds takes the running-maximum form for that segment.
// (The scan over segments in this form measured no faster: it saves exponentials and needs two more rounds of shuffles.)
constexpr float kSpan = 40.f, kBonus = 20.f;
struct Range {
    float lo, hi;
};
__device__ __forceinline__ Range range_of(const float (&k)[L], int n) {
    Range r = {k[0], k[0]};
#pragma unroll
    for (int i = 1; i < L; ++i)
        if (i < n) { r.lo = fminf(r.lo, k[i]); r.hi = fmaxf(r.hi, k[i]); }
    return r;
}
// the start state joins the range (an empty one has no exponent): true if plain weights relative to r.hi serve
__device__ __forceinline__ bool join(Range& r, const Sum& s) {
    if (s.q != 0.f) { r.lo = fminf(r.lo, s.o); r.hi = fmaxf(r.hi, s.o); }
    return r.hi - r.lo <= kSpan;
}

template <int S>
struct ScanBuf {
    float x[3][S][33];
    float w[32];
    float carry[3][32];
};

// Start states of the S segments of a tile from their local sums and the state carried in from the tile before (in walking
// order: REV walks the segments from S-1 down).  Called by all warps; leaves the carried state after the tile in `buf`.
template <int S, bool REV>
__device__ __forceinline__ Sum scan_segments(ScanBuf<S>& buf, Sum local, int warp, int lane) {
    buf.x[0][warp][lane] = local.p; buf.x[1][warp][lane] = local.q; buf.x[2][warp][lane] = local.o;
    __syncthreads();
    {   // this thread: channel ch, segment number i in walking order
        const int ch = warp * (32 / S) + lane / S, i = lane & (S - 1), seg = REV ? S - 1 - i : i;
        const float lw = L * buf.w[ch];
        Sum s = {buf.x[0][seg][ch], buf.x[1][seg][ch], buf.x[2][seg][ch]};
        const Sum c = {buf.carry[0][ch], buf.carry[1][ch], buf.carry[2][ch]};
        if (i == 0) s = after(c, lw, s);
#pragma unroll
        for (int m = 1; m < S; m <<= 1) {   // inclusive: s covers up to 2 m segments after the step
            Sum f;
            f.p = __shfl_up_sync(0xffffffffu, s.p, m, S);
            f.q = __shfl_up_sync(0xffffffffu, s.q, m, S);
            f.o = __shfl_up_sync(0xffffffffu, s.o, m, S);
            const Sum t = after(f, m * lw, s);
            if (i >= m) s = t;
        }
        Sum e;                               // exclusive: the state before this segment
        e.p = __shfl_up_sync(0xffffffffu, s.p, 1, S);
        e.q = __shfl_up_sync(0xffffffffu, s.q, 1, S);
        e.o = __shfl_up_sync(0xffffffffu, s.o, 1, S);
        if (i == 0) e = c;
        __syncwarp();
        buf.x[0][seg][ch] = e.p; buf.x[1][seg][ch] = e.q; buf.x[2][seg][ch] = e.o;
        if (i == S - 1) { buf.carry[0][ch] = s.p; buf.carry[1][ch] = s.q; buf.carry[2][ch] = s.o; }
    }
    __syncthreads();
    return Sum{buf.x[0][warp][lane], buf.x[1][warp][lane], buf.x[2][warp][lane]};
}

// Start states of the segments, (p, q, o) of 32 channels each: segment s >= 1 of batch row b at p[b * row + (s - 1) * seg + i * C + c].
// (Segment 0 starts empty.)  Either a buffer of their own, or parked in an output the reverse pass overwrites later.
struct States {
    float* p;
    i64 row, seg;
};

struct Place {         // what a block works on
    int b, c;
    bool live;
};
__device__ __forceinline__ Place place(int C, int lane) {
    const int groups = (C + 31) / 32, b = blockIdx.x / groups, c = (blockIdx.x - b * groups) * 32 + lane;
    return Place{b, min(c, C - 1), c < C};
}

// A segment of n tokens from state s in the running-maximum form: y (if y_ is given) and the state behind it.
__device__ __noinline__ Sum forward_running_max(Sum s, int n, float w, float u, const float* k_, const float* v_, float* y_, int C) {
    for (int i = 0; i < n; ++i) {
        const float k = k_[(i64)i * C], v = v_[(i64)i * C];
        if (y_ != nullptr) {
            const Pair e = softpair(s.o, u + k);
            y_[(i64)i * C] = (e.a * s.p + e.b * v) / (e.a * s.q + e.b);
        }
        s = after(s, w, Sum{v, 1.f, k});
    }
    return s;
}

template <int S, bool Y>
__global__ void __launch_bounds__(32 * S) wkv4_forward_kernel(int T, int C, const float* __restrict__ w_, int w_raw, const float* __restrict__ u_,
                                                              const float* __restrict__ k_, const float* __restrict__ v_,
                                                              float* __restrict__ y_, States st, unsigned* counters) {
    __shared__ ScanBuf<S> buf;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const Place at = place(C, lane);
    const i64 off = (i64)at.b * T * C + at.c;
    const float w = w_raw ? -expf(w_[at.c]) : w_[at.c], u = u_[at.c], ew = expf(w), eu = expf(u);
    const bool bonus_ok = fabsf(u) <= kBonus;
    if (counters != nullptr && threadIdx.x == 0 && at.b == 0) counters[blockIdx.x] = 0;   // for the backward
    if (warp == 0) { buf.w[lane] = w; buf.carry[0][lane] = 0.f; buf.carry[1][lane] = 0.f; buf.carry[2][lane] = kNegInf; }
    float kn[L], vn[L];
    auto fetch = [&](int t0) {
        const i64 o = off + (i64)t0 * C;
        const float *kp = k_ + o, *vp = v_ + o;
#pragma unroll
        for (int i = 0; i < L; ++i) {
            const bool in = t0 + i < T;
            kn[i] = in ? kp[i * C] : 0.f;
            vn[i] = in ? vp[i * C] : 0.f;
        }
    };
    fetch(warp * L);
    for (int t0 = warp * L; t0 - warp * L < T; t0 += S * L) {
        float k[L], v[L];
#pragma unroll
        for (int i = 0; i < L; ++i) { k[i] = kn[i]; v[i] = vn[i]; }
        fetch(t0 + S * L);   // the next tile's loads are in flight during this tile's math
        const int n = T - t0;
        const bool full = n >= L;   // whole segments have their own loops: no test per token
        Range rg = full ? range_of(k, L) : range_of(k, n);
        Sum s = {0.f, 0.f, kNegInf};
        float e[L], base = rg.hi;
        const bool plain = __all_sync(0xffffffffu, bonus_ok && rg.hi - rg.lo <= kSpan);
        if (plain) {
#pragma unroll
            for (int i = 0; i < L; ++i) e[i] = expf(k[i] - rg.hi);
            if (full) {
#pragma unroll
                for (int i = 0; i < L; ++i) { s.p = fmaf(s.p, ew, e[i] * v[i]); s.q = fmaf(s.q, ew, e[i]); }
            } else {
#pragma unroll
                for (int i = 0; i < L; ++i)
                    if (i < n) { s.p = fmaf(s.p, ew, e[i] * v[i]); s.q = fmaf(s.q, ew, e[i]); }
            }
            if (n > 0) s.o = rg.hi;
        } else {
            s = forward_running_max(s, min(n, L), w, u, k_ + off + (i64)t0 * C, v_ + off + (i64)t0 * C, nullptr, C);
        }
        s = scan_segments<S, false>(buf, s, warp, lane);
        if (st.p != nullptr && t0 > 0 && n > 0 && at.live) {
            float* p = st.p + at.b * st.row + (t0 / L - 1) * st.seg + at.c;
            p[0] = s.p; p[C] = s.q; p[2 * (i64)C] = s.o;
        }
        if (Y && plain && __all_sync(0xffffffffu, join(rg, s))) {
            const float fs = s.q != 0.f ? expf(s.o - rg.hi) : 0.f, fk = expf(base - rg.hi);
            float p = s.p * fs, q = s.q * fs;
            float* yp = y_ + off + (i64)t0 * C;
            auto token = [&](int i) {
                const float x = e[i] * fk, xu = x * eu;
                if (at.live) yp[i * C] = fmaf(xu, v[i], p) / (q + xu);
                p = fmaf(p, ew, x * v[i]);
                q = fmaf(q, ew, x);
            };
            if (full) {
#pragma unroll
                for (int i = 0; i < L; ++i) token(i);
            } else {
#pragma unroll
                for (int i = 0; i < L; ++i)
                    if (i < n) token(i);
            }
        } else if (Y && at.live) {
            forward_running_max(s, min(n, L), w, u, k_ + off + (i64)t0 * C, v_ + off + (i64)t0 * C, y_ + off + (i64)t0 * C, C);
        }
    }
}

// A segment of n tokens in reverse in the running-maximum form: gk, gv from its start state and the adjoint G behind it; returns
// its part of dL/dw.
__device__ __noinline__ float reverse_running_max(Sum start, Sum G, int n, float w, float u, const float* k_, const float* v_, const float* g_,
                                                  float* gk_, float* gv_, int C, bool live) {
    Sum before[L];
    float ld[L], y[L], A[L], gw = 0.f;
    for (int i = 0; i < n; ++i) {
        const float k = k_[(i64)i * C], v = v_[(i64)i * C];
        before[i] = start;
        const Pair x = softpair(start.o, u + k);
        const float den = x.a * start.q + x.b, iden = 1.f / den;
        y[i] = (x.a * start.p + x.b * v) * iden;
        ld[i] = x.m + logf(den);
        A[i] = g_[(i64)i * C] * x.b * iden;
        start = after(start, w, Sum{v, 1.f, k});
    }
    for (int i = n - 1; i >= 0; --i) {
        const float k = k_[(i64)i * C], v = v_[(i64)i * C], g = g_[(i64)i * C], Bk = expf(k + G.o);
        gw = fmaf(expf(w + G.o + before[i].o), fmaf(G.p, before[i].p, G.q * before[i].q), gw);
        if (live) {
            gk_[(i64)i * C] = A[i] * (v - y[i]) + Bk * fmaf(G.p, v, G.q);
            gv_[(i64)i * C] = fmaf(Bk, G.p, A[i]);
        }
        G = after(G, w, Sum{g, -g * y[i], -ld[i]});
    }
    return gw;
}

// gw, gu: per batch row (row stride gstride), added to when `accumulate`.  With `sum_` (2,C) the last block of a channel group to
// finish adds the rows up in order (counters[group] counts the others and is left at zero): no launch for it.
template <int S>
__global__ void __launch_bounds__(32 * S, S == 8 ? 3 : 1) wkv4_backward_kernel(int T, int C, const float* __restrict__ w_, int w_raw,
                                                                       const float* __restrict__ u_, const float* __restrict__ k_,
                                                                       const float* __restrict__ v_, const float* __restrict__ gy_,
                                                                       States st, float* __restrict__ gw_, float* __restrict__ gu_,
                                                                       i64 gstride, int accumulate, float* gk_, float* gv_, int B,
                                                                       float* sum_, unsigned* counters) {
    __shared__ ScanBuf<S> buf;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const Place at = place(C, lane);
    const i64 off = (i64)at.b * T * C + at.c;
    const float w = w_raw ? -expf(w_[at.c]) : w_[at.c], u = u_[at.c], ew = expf(w), eu = expf(u);
    const bool bonus_ok = fabsf(u) <= kBonus;
    if (warp == 0) { buf.w[lane] = w; buf.carry[0][lane] = 0.f; buf.carry[1][lane] = 0.f; buf.carry[2][lane] = kNegInf; }
    float gw = 0.f, gw_plain = 0.f, gu = 0.f;   // gw_plain: without the factor e^w
    for (int t0 = (T - 1) / (S * L) * (S * L) + warp * L; t0 >= 0; t0 -= S * L) {
        const int n = T - t0;
        const bool full = n >= L;
        const i64 o0 = off + (i64)t0 * C;
        float k[L], v[L], g[L];
        {
            const float *kp = k_ + o0, *vp = v_ + o0, *gp = gy_ + o0;
#pragma unroll
            for (int i = 0; i < L; ++i) {
                const bool in = i < n;
                k[i] = in ? kp[i * C] : 0.f; v[i] = in ? vp[i * C] : 0.f; g[i] = in ? gp[i * C] : 0.f;
            }
        }
        Sum s = {0.f, 0.f, kNegInf};
        if (t0 > 0 && n > 0) {
            const float* p = st.p + at.b * st.row + (t0 / L - 1) * st.seg + at.c;
            s = Sum{p[0], p[C], p[2 * (i64)C]};
        }
        const Sum start = s;
        Range rg = full ? range_of(k, L) : range_of(k, n);
        const bool plain = __all_sync(0xffffffffu, bonus_ok && join(rg, s));
        // forward inside the segment: the running sums before each token, y, and the token's term h (1, -y) of the adjoint (all in
        // units of the largest weight); then the adjoint that the segment adds by itself
        float bp[L], bq[L], y[L], h[L], e[L];
        Sum G = {0.f, 0.f, kNegInf};
        if (plain) {
            const float fs = s.q != 0.f ? expf(s.o - rg.hi) : 0.f;
            s.p *= fs; s.q *= fs;
#pragma unroll
            for (int i = 0; i < L; ++i) {
                e[i] = expf(k[i] - rg.hi);
                const float xu = e[i] * eu, iden = 1.f / (s.q + xu);
                bp[i] = s.p; bq[i] = s.q;
                y[i] = fmaf(xu, v[i], s.p) * iden;
                h[i] = g[i] * iden;
                if (i < n) gu = fmaf(h[i] * xu, v[i] - y[i], gu);   // (beyond the end k is 0, which may be far outside of the range)
                s.p = fmaf(s.p, ew, e[i] * v[i]);
                s.q = fmaf(s.q, ew, e[i]);
            }
            if (full) {
#pragma unroll
                for (int i = L - 1; i >= 0; --i) { G.p = fmaf(G.p, ew, h[i]); G.q = fmaf(G.q, ew, -h[i] * y[i]); }
            } else {
#pragma unroll
                for (int i = L - 1; i >= 0; --i)
                    if (i < n) { G.p = fmaf(G.p, ew, h[i]); G.q = fmaf(G.q, ew, -h[i] * y[i]); }
            }
            if (n > 0) G.o = -rg.hi;
        } else {
            // running-maximum form; y and log den are rebuilt by the reverse walk
#pragma unroll
            for (int i = 0; i < L; ++i) {
                const Pair x = softpair(s.o, u + k[i]);
                const float den = x.a * s.q + x.b, iden = 1.f / den;
                y[i] = (x.a * s.p + x.b * v[i]) * iden;
                gu = fmaf(g[i] * x.b * iden, v[i] - y[i], gu);
                h[i] = x.m + logf(den);
                s = after(s, w, Sum{v[i], 1.f, k[i]});
            }
#pragma unroll
            for (int i = L - 1; i >= 0; --i)
                if (i < n) G = after(G, w, Sum{g[i], -g[i] * y[i], -h[i]});
        }
        G = scan_segments<S, true>(buf, G, warp, lane);
        const bool empty = G.p == 0.f && G.q == 0.f;
        if (plain && __all_sync(0xffffffffu, empty || fabsf(G.o + rg.hi) <= kSpan)) {
            const float f = empty ? 0.f : expf(G.o + rg.hi);
            float gp = G.p * f, gq = G.q * f;
            float *gkp = gk_ + o0, *gvp = gv_ + o0;
            auto token = [&](int i) {
                const float A = h[i] * e[i] * eu;
                gw_plain = fmaf(gp, bp[i], fmaf(gq, bq[i], gw_plain));
                if (at.live) {
                    gkp[i * C] = fmaf(A, v[i] - y[i], e[i] * fmaf(gp, v[i], gq));
                    gvp[i * C] = fmaf(e[i], gp, A);
                }
                gp = fmaf(gp, ew, h[i]);
                gq = fmaf(gq, ew, -h[i] * y[i]);
            };
            if (full) {
#pragma unroll
                for (int i = L - 1; i >= 0; --i) token(i);
            } else {
#pragma unroll
                for (int i = L - 1; i >= 0; --i)
                    if (i < n) token(i);
            }
        } else {
            gw += reverse_running_max(start, G, min(n, L), w, u, k_ + off + (i64)t0 * C, v_ + off + (i64)t0 * C, gy_ + off + (i64)t0 * C,
                                      gk_ + off + (i64)t0 * C, gv_ + off + (i64)t0 * C, C, at.live);
        }
    }
    gw = fmaf(ew, gw_plain, gw);
    __syncthreads();
    buf.x[0][warp][lane] = gw; buf.x[1][warp][lane] = gu;
    __syncthreads();
    if (warp == 0 && at.live) {
        gw = 0.f; gu = 0.f;
#pragma unroll
        for (int i = 0; i < S; ++i) { gw += buf.x[0][i][lane]; gu += buf.x[1][i][lane]; }
        gw *= w;   // the chain rule through w = -exp(time_decay) is applied here, as the reference does
        float *pw = gw_ + at.b * gstride + at.c, *pu = gu_ + at.b * gstride + at.c;
        if (accumulate) { gw += *pw; gu += *pu; }
        *pw = gw; *pu = gu;
    }
    if (sum_ == nullptr || warp != 0) return;
    const int group = blockIdx.x % ((C + 31) / 32);
    __threadfence();
    __syncwarp();
    unsigned before = 0;
    if (lane == 0) before = atomicAdd(counters + group, 1u);
    if (__shfl_sync(0xffffffffu, before, 0) != (unsigned)(B - 1)) return;
    __threadfence();
    if (lane == 0) counters[group] = 0;
    if (!at.live) return;
    gw = 0.f; gu = 0.f;
#pragma unroll 4
    for (int b = 0; b < B; ++b) { gw += __ldcg(gw_ + b * gstride + at.c); gu += __ldcg(gu_ + b * gstride + at.c); }
    sum_[at.c] = gw; sum_[C + at.c] = gu;
}

// S: the fewest blocks get the most warps (32 channel groups are a fifth of the SMs); with more groups than SMs short tiles,
// so that several blocks share an SM.  No more segments than the sequence has.
int pick_segments(int B, int T, int C, int most) {
    const i64 groups = (i64)B * ((C + 31) / 32);
    const int sms = sm_count();
    int S = groups <= sms ? 32 : groups <= 2 * sms ? 16 : 8;
    while (S > 8 && (S > most || (S / 2) * L >= T)) S /= 2;
    return S;
}
i64 group_count(int B, int C) { return (i64)B * ((C + 31) / 32); }

int forward(int B, int T, int C, const float* w, int w_raw, const float* u, const float* k, const float* v, float* y, States st,
            unsigned* counters, cudaStream_t s) {
    const unsigned grid = (unsigned)group_count(B, C);
#define RWKV_GO(SEG)                                                                                                    \
    do {                                                                                                                \
        if (y != nullptr) wkv4_forward_kernel<SEG, true><<<grid, 32 * SEG, 0, s>>>(T, C, w, w_raw, u, k, v, y, st, counters); \
        else wkv4_forward_kernel<SEG, false><<<grid, 32 * SEG, 0, s>>>(T, C, w, w_raw, u, k, v, y, st, counters); \
    } while (0)
    switch (pick_segments(B, T, C, 32)) {
        case 32: RWKV_GO(32); break;
        case 16: RWKV_GO(16); break;
        default: RWKV_GO(8); break;
    }
#undef RWKV_GO
    return check_launch("wkv4_forward");
}

int backward(int B, int T, int C, const float* w, int w_raw, const float* u, const float* k, const float* v, const float* gy, States st,
             float* gw, float* gu, i64 gstride, int accumulate, float* gk, float* gv, float* sum, unsigned* counters, cudaStream_t s) {
    const unsigned grid = (unsigned)group_count(B, C);
    if (pick_segments(B, T, C, 16) == 16)
        wkv4_backward_kernel<16><<<grid, 512, 0, s>>>(T, C, w, w_raw, u, k, v, gy, st, gw, gu, gstride, accumulate, gk, gv, B, sum, counters);
    else
        wkv4_backward_kernel<8><<<grid, 256, 0, s>>>(T, C, w, w_raw, u, k, v, gy, st, gw, gu, gstride, accumulate, gk, gv, B, sum, counters);
    return check_launch("wkv4_backward");
}

States saved_states(float* p, int T, int C) {
    const i64 nseg = (T + L - 1) / L;
    return States{p, (nseg - 1) * 3 * C, 3 * (i64)C};
}

unsigned* saved_counters(void* p, int B, int T, int C) {   // behind the states
    return static_cast<unsigned*>(p) + (size_t)B * ((T + L - 1) / L - 1) * 3 * C;
}

}  // namespace

}  // namespace rwkvb200

using namespace rwkvb200;

static int check_wkv4(const char* what, int B, int T, int C) {
    RWKV_REQUIRE(B > 0 && T > 0 && C > 0, RWKVB200_EINVAL, "%s: B=%d T=%d C=%d must be positive", what, B, T, C);
    RWKV_REQUIRE((i64)B * C < (1ll << 31), RWKVB200_EINVAL, "%s: B*C too large", what);
    return RWKVB200_OK;
}

extern "C" int rwkvb200_wkv4_forward(int B, int T, int C, const float* w, const float* u, const float* k,
                                     const float* v, float* y, void* stream) {
    if (int e = check_wkv4("wkv4_forward", B, T, C)) return e;
    RWKV_NOTNULL(w); RWKV_NOTNULL(u); RWKV_NOTNULL(k); RWKV_NOTNULL(v); RWKV_NOTNULL(y);
    return forward(B, T, C, w, 0, u, k, v, y, States{nullptr, 0, 0}, nullptr, as_stream(stream));
}

extern "C" int rwkvb200_wkv4_backward(int B, int T, int C, const float* w, const float* u, const float* k,
                                      const float* v, const float* gy, float* gw, float* gu, float* gk,
                                      float* gv, void* stream) {
    if (int e = check_wkv4("wkv4_backward", B, T, C)) return e;
    RWKV_NOTNULL(w); RWKV_NOTNULL(u); RWKV_NOTNULL(k); RWKV_NOTNULL(v); RWKV_NOTNULL(gy);
    RWKV_NOTNULL(gw); RWKV_NOTNULL(gu); RWKV_NOTNULL(gk); RWKV_NOTNULL(gv);
    // A states-only forward pass parks the start state of every segment in the gk slots of the segment before it; the
    // reverse pass reads a segment's state before it writes the gk of the one before.
    const States st = {gk, (i64)T * C, (i64)L * C};
    if (T > L)
        if (int e = forward(B, T, C, w, 0, u, k, v, nullptr, st, nullptr, as_stream(stream))) return e;
    return backward(B, T, C, w, 0, u, k, v, gy, st, gw, gu, C, 1, gk, gv, nullptr, nullptr, as_stream(stream));
}

extern "C" size_t rwkvb200_wkv4_saved_bytes(int B, int T, int C) {
    if (B <= 0 || T <= 0 || C <= 0) return 0;
    return ((size_t)B * ((T + L - 1) / L - 1) * 3 * C + (C + 31) / 32) * sizeof(float);   // states, and a counter per channel group
}

extern "C" int rwkvb200_wkv4_train_forward(int B, int T, int C, const float* w_raw, const float* u, const float* k, const float* v,
                                           float* y, void* saved, void* stream) {
    if (int e = check_wkv4("wkv4_train_forward", B, T, C)) return e;
    RWKV_NOTNULL(w_raw); RWKV_NOTNULL(u); RWKV_NOTNULL(k); RWKV_NOTNULL(v); RWKV_NOTNULL(y); RWKV_NOTNULL(saved);
    return forward(B, T, C, w_raw, 1, u, k, v, y, saved_states(static_cast<float*>(saved), T, C), saved_counters(saved, B, T, C), as_stream(stream));
}

extern "C" int rwkvb200_wkv4_train_backward(int B, int T, int C, const float* w_raw, const float* u, const float* k, const float* v,
                                            const float* gy, const void* saved, float* gwu, float* partial, float* gk, float* gv,
                                            void* stream) {
    if (int e = check_wkv4("wkv4_train_backward", B, T, C)) return e;
    RWKV_NOTNULL(w_raw); RWKV_NOTNULL(u); RWKV_NOTNULL(k); RWKV_NOTNULL(v); RWKV_NOTNULL(gy); RWKV_NOTNULL(saved);
    RWKV_NOTNULL(gwu); RWKV_NOTNULL(gk); RWKV_NOTNULL(gv);
    RWKV_REQUIRE(B == 1 || partial != nullptr, RWKVB200_ENULL, "wkv4_train_backward: partial is NULL");
    float* p = B == 1 ? gwu : partial;
    const States st = saved_states(static_cast<float*>(const_cast<void*>(saved)), T, C);
    return backward(B, T, C, w_raw, 1, u, k, v, gy, st, p, p + C, 2 * (i64)C, 0, gk, gv, B == 1 ? nullptr : gwu,
                    saved_counters(const_cast<void*>(saved), B, T, C), as_stream(stream));
}
