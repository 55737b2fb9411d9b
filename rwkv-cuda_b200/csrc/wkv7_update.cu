// RWKV-7 inference, head size 64, fp32 or bf16 activations, fp32 arithmetic and state: advances the state of every
// (batch, head) unit in place by T tokens.  Two kernels:
//
// wkv7_decode_kernel, T = 1.  The state of a unit is read once and written once (32 KB, for 7 vectors of 64 elements), so
// HBM bounds it.  128 threads per unit, 16 lanes x float4 on a row of the state: every access of a warp is 512
// consecutive bytes and 8 of them are in flight per thread.  B = 128, H = 32 on a B200: 140 us for the general-shape
// kernel (one thread per row: 256-byte strides), 25 us here (5.5 TB/s).
//
// wkv7_rows_kernel, T > 1 (prompts of any length).  The recurrence of one value row
//     sa_t = S_{t-1}.a_t      S_t = S_{t-1} d_t + sa_t b_t + v_t k_t      y_t = S_t.r_t
// needs nothing of the other 63 rows, so a unit is spread over 1 to 4 blocks; what bounds a launch with few units is the
// chain from one dot product over 64 keys, with its reduction over lanes, to the next, and, with many rows on an SM, the
// shared-memory reads of the tokens' vectors (2 / RPT wavefronts per row and vector whatever the lane split).
// So four tokens are one step.  With W_t = d_0 .. d_t inside the step (t = 0 .. 3)
//     a~_t = a_t W_{t-1}    r~_t = r_t W_t    b^_s = b_s d_{s+1} .. d_3    k^_s = k_s d_{s+1} .. d_3
//     sa_t = S.a~_t + sum_{s<t} sa_s Ub[s,t] + v_s Uk[s,t]         Ub[s,t] = b_s.(a_t d_{s+1} .. d_{t-1}), Uk with k_s
//     y_t  = S.r~_t + sum_{s<=t} sa_s Rb[s,t] + v_s Rk[s,t]        Rb[s,t] = b_s.(r_t d_{s+1} .. d_t), Rk with k_s
//     S   <- S W_3 + sum_s sa_s b^_s + v_s k^_s
// the eight dot products of a row are reduced together (8 shuffles, not 4 per token), 17 vectors are read instead of 20, and the
// chain has one reduction per four tokens.  NCW warps compute; NSW warps stage, a step each: they make the scaled vectors (products of
// decays are carried as sums of two numbers: a vector is rounded once) and the 32 scalars of a step, which all rows share.
// One sequence of 1999 tokens, 32 heads: 2010 us for the general-shape kernel, 213 us with a token as a step, 209 us here; 128 units
// 428 -> 394 us, 256 units 852 -> 700 us.  A step takes 790 clocks where a unit has four SMs: 350 of the shared-memory reads, the
// rest 430 instructions per scheduler, of one warp that computes and one or two that stage (four staging warps 209 us, eight 201; with
// more rows per block eight were slower: 128 units 411 us).
// Errors against fp64 (T 1999, H 8, of the norm): state 8.3e-8, y 1.11e-7; a token as a step 8.7e-8 and 1.12e-7.  Most of the state is of the last
// few tokens, and where all eight terms of a step went onto it one by one, each was rounded at its full size (9.3e-8, 1.14e-7); so
// the four of sa are summed first (one more instruction per pair: 256 units 670 -> 690).  What is not finite goes token by token: rows_again.
#include "common.cuh"
#include "packed.cuh"
#include "wkv7_dispatch.cuh"

namespace rwkvb200 {
namespace {

constexpr int kN = 64;
constexpr float kWScale7 = -0.6065306597126334f;  // -exp(-1/2)

__device__ __forceinline__ float decay7(float w) { return __expf(kWScale7 * __fdividef(1.f, 1.f + __expf(-w))); }

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const bf16* p) {
    const uint2 x = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(x.x << 16), __uint_as_float(x.x & 0xffff0000u), __uint_as_float(x.y << 16), __uint_as_float(x.y & 0xffff0000u));
}

// Sums of v[0..7] over the 16 lanes of a half warp in 8 shuffles: lane x ends with the sum of v[x >> 1].
__device__ __forceinline__ float reduce8_over16(float (&v)[8], int lane) {
#pragma unroll
    for (int m = 8, n = 4; n >= 1; m >>= 1, n >>= 1) {
        const bool up = (lane & m) != 0;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

template <typename E>
__global__ void __launch_bounds__(128) wkv7_decode_kernel(float* __restrict__ state, const E* __restrict__ r_, const E* __restrict__ w_,
                                                          const E* __restrict__ k_, const E* __restrict__ v_, const E* __restrict__ a_,
                                                          const E* __restrict__ b_, E* __restrict__ y_) {
    const int tid = threadIdx.x, lane = tid & 31, row0 = tid >> 4;
    const i64 unit = blockIdx.x;
    float* st = state + unit * kN * kN + tid * 4;
    const i64 vec = unit * kN, key = vec + (tid & 15) * 4;
    float4 S[8];   // S[i]: row 8 i + row0, keys 4 (tid & 15) ..
#pragma unroll
    for (int i = 0; i < 8; ++i) S[i] = *reinterpret_cast<const float4*>(st + i * 512);
    const float4 a = load4(a_ + key), b = load4(b_ + key), k = load4(k_ + key), r = load4(r_ + key), w = load4(w_ + key);
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = to_f(v_[vec + 8 * i + row0]);
    const float4 d = make_float4(decay7(w.x), decay7(w.y), decay7(w.z), decay7(w.w));
    float p[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) p[i] = fmaf(S[i].w, a.w, fmaf(S[i].z, a.z, fmaf(S[i].y, a.y, S[i].x * a.x)));
    const float sum = reduce8_over16(p, lane);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float sa = __shfl_sync(0xffffffffu, sum, (lane & 16) + 2 * i);
        S[i].x = fmaf(S[i].x, d.x, fmaf(sa, b.x, k.x * v[i]));
        S[i].y = fmaf(S[i].y, d.y, fmaf(sa, b.y, k.y * v[i]));
        S[i].z = fmaf(S[i].z, d.z, fmaf(sa, b.z, k.z * v[i]));
        S[i].w = fmaf(S[i].w, d.w, fmaf(sa, b.w, k.w * v[i]));
        *reinterpret_cast<float4*>(st + i * 512) = S[i];
        p[i] = fmaf(S[i].w, r.w, fmaf(S[i].z, r.z, fmaf(S[i].y, r.y, S[i].x * r.x)));
    }
    const float y = reduce8_over16(p, lane);
    if ((lane & 1) == 0) y_[vec + 8 * ((lane & 15) >> 1) + row0] = from_f<E>(y);
}

// ---- prompts ----------------------------------------------------------------------------------------------
// The 64 / LG keys of lane x of a row (LG = 8 or 16 lanes).  In shared memory the first four of every eight keys come
// first, then the other four, so that eight lanes read and write 128 consecutive bytes: staged_at(key) is the place.
template <int LG>
__device__ __forceinline__ int first_key(int x) { return LG == 8 ? 8 * x : 8 * (x & 7) + ((x & 8) >> 1); }
template <int LG>
struct Keys { f2 x[32 / LG]; };
template <int LG>
__device__ __forceinline__ Keys<LG> load_keys(const float* row, int x) {
    Keys<LG> k;
#pragma unroll
    for (int h = 0; h < 16 / LG; ++h) {
        const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(row + 32 * h + 4 * x);
        k.x[2 * h] = p.x; k.x[2 * h + 1] = p.y;
    }
    return k;
}
template <int LG>
__device__ __forceinline__ float dot_keys(const f2 (&s)[32 / LG], const Keys<LG>& a) {
    f2 acc = mul2(s[0], a.x[0]);
#pragma unroll
    for (int e = 1; e < 32 / LG; ++e) acc = fma2(s[e], a.x[e], acc);
    return sum2(acc);
}
constexpr int kQ = 4;   // tokens of a step
// The scaled vectors of a step, the products of its decays (w), its values, and the scalars of the steps inside it: b, k of token s
// against a of token t (s < t) at ((t - 1) t / 2 + s) * 2, then against r of token t (s <= t, nothing above) at 12 + 8 t + 2 s.
struct __align__(16) Step { float a[kQ][kN], r[kQ][kN], b[kQ][kN], k[kQ][kN], w[kN], v[kQ][kN], u[12 + 8 * kQ]; int odd; };
template <int NSW>
struct __align__(16) Staged { Step s[NSW]; };   // a step per staging warp

// Two neighbouring elements, as loaded and decoded
template <typename E> struct Pair2;
template <> struct Pair2<bf16> { uint32_t x; };
template <> struct Pair2<float> { float2 x; };
template <typename E>
__device__ __forceinline__ Pair2<E> load2(const E* p, bool in) {
    Pair2<E> r;
    if constexpr (sizeof(E) == 2) r.x = in ? __ldg(reinterpret_cast<const uint32_t*>(p)) : 0u;
    else r.x = in ? __ldg(reinterpret_cast<const float2*>(p)) : make_float2(0.f, 0.f);
    return r;
}
__device__ __forceinline__ float2 decode2(Pair2<bf16> p) { return make_float2(__uint_as_float(p.x << 16), __uint_as_float(p.x & 0xffff0000u)); }
__device__ __forceinline__ float2 decode2(Pair2<float> p) { return p.x; }
__device__ __forceinline__ float2 times(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
struct Exact2 { float2 hi, lo; };   // hi + lo, for two keys
__device__ __forceinline__ float2 times(float2 a, Exact2 b) { return make_float2(fmaf(a.x, b.hi.x, a.x * b.lo.x), fmaf(a.y, b.hi.y, a.y * b.lo.y)); }
__device__ __forceinline__ Exact2 times(Exact2 a, float2 b) {
    const float2 h = times(a.hi, b);
    return Exact2{h, make_float2(fmaf(a.lo.x, b.x, fmaf(a.hi.x, b.x, -h.x)), fmaf(a.lo.y, b.y, fmaf(a.hi.y, b.y, -h.y)))};
}
__device__ __forceinline__ float dot2(float2 a, float2 b) { return fmaf(a.y, b.y, a.x * b.x); }
__device__ __forceinline__ void prefetch_l2(const void* p) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(__cvta_generic_to_global(p)));
}
// named barriers ID + odd (constants: a barrier number in a register makes the block reserve all sixteen)
template <int ID, int NTH>
__device__ __forceinline__ void bar_sync(int odd) {
    if (odd) asm volatile("bar.sync %0, %1;" ::"n"(ID + 1), "n"(NTH) : "memory");
    else asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(NTH) : "memory");
}
template <int ID, int NTH>
__device__ __forceinline__ void bar_arrive(int odd) {
    if (odd) asm volatile("bar.arrive %0, %1;" ::"n"(ID + 1), "n"(NTH) : "memory");
    else asm volatile("bar.arrive %0, %1;" ::"n"(ID), "n"(NTH) : "memory");
}
// Sums of v[0..7] over LG lanes: lane x ends with the sum of v[x >> 1] (16 lanes) or v[x] (8 lanes).
template <int LG>
__device__ __forceinline__ float reduce8_over(float (&v)[8], int x) {
#pragma unroll
    for (int m = LG / 2, n = 4; n >= 1; m >>= 1, n >>= 1) {
        const bool up = (x & m) != 0;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
        }
    }
    return LG == 16 ? v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1) : v[0];
}
// RPT neighbouring outputs
template <typename E, int RPT>
__device__ __forceinline__ void store_rows(E* p, const float (&y)[RPT]) {
    if constexpr (sizeof(E) == 2) {
        uint32_t w[RPT / 2];
#pragma unroll
        for (int i = 0; i < RPT / 2; ++i) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(y[2 * i], y[2 * i + 1]);
            w[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
        if constexpr (RPT == 2) *reinterpret_cast<uint32_t*>(p) = w[0];
        else *reinterpret_cast<uint2*>(p) = make_uint2(w[0], w[1]);
    } else {
        if constexpr (RPT == 2) *reinterpret_cast<float2*>(p) = make_float2(y[0], y[1]);
        else *reinterpret_cast<float4*>(p) = make_float4(y[0], y[1], y[2], y[3]);
    }
}

// sums that are 0 unless one of the values is not finite
__device__ __forceinline__ void check(float& bad, float x) { bad = fmaf(x, 0.f, bad); }

// The rows of a warp once more, token by token from the state in memory: with values that are not finite the sums over four tokens are
// others than token by token (infinities of both signs meet, parts of a product are infinity times 0), and NaN would stand where the
// recurrence gives an infinity.  S_t = G_t + sa_t b_t with G_t = S_{t-1} d_t + v_t k_t, and sa_{t+1} = G_t.a_{t+1} + sa_t (b_t.a_{t+1}).
// What is a number in both forms stays as it is (other: the state by steps of four): in what order it was summed does not depend on
// a value beyond its reach.
template <typename E, int LG, int RPT>
__device__ __noinline__ void rows_again(int T, int C, i64 base, int row0, int x, float* st, const E* r_, const E* w_, const E* k_, const E* v_,
                                        const E* a_, const E* b_, E* y_, const float (&other)[RPT][64 / LG]) {
    constexpr int K = 64 / LG;
    auto sum = [](float p) {
#pragma unroll
        for (int m = 1; m < LG; m <<= 1) p += __shfl_xor_sync(0xffffffffu, p, m);
        return p;
    };
    const i64 key = base + first_key<LG>(x);
    float S[RPT][K], sa[RPT];
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        float p = 0.f;
#pragma unroll
        for (int j = 0; j < K; ++j) { S[i][j] = st[i * kN + j]; p = fmaf(S[i][j], to_f(a_[key + j]), p); }
        sa[i] = sum(p);
    }
    for (int t = 0; t < T; ++t) {
        const i64 o = (i64)t * C;
        float d[K], k[K], b[K], r[K], an[K], beta = 0.f;
#pragma unroll
        for (int j = 0; j < K; ++j) {
            d[j] = decay7(to_f(w_[o + key + j])); k[j] = to_f(k_[o + key + j]); b[j] = to_f(b_[o + key + j]); r[j] = to_f(r_[o + key + j]);
            an[j] = t + 1 < T ? to_f(a_[o + C + key + j]) : 0.f;
            beta = fmaf(b[j], an[j], beta);
        }
        beta = sum(beta);
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            const float v = to_f(v_[o + base + row0 + i]);
            float z = 0.f, y = 0.f;
#pragma unroll
            for (int j = 0; j < K; ++j) {
                S[i][j] = fmaf(S[i][j], d[j], k[j] * v);
                z = fmaf(S[i][j], an[j], z);
                S[i][j] = fmaf(sa[i], b[j], S[i][j]);
                y = fmaf(S[i][j], r[j], y);
            }
            y = sum(y);
            sa[i] = fmaf(sa[i], beta, sum(z));
            E* p = y_ + o + base + row0 + i;
            if (x == 0 && !(isfinite(y) && isfinite(to_f(*p)))) *p = from_f<E>(y);
        }
    }
#pragma unroll
    for (int i = 0; i < RPT; ++i)
#pragma unroll
        for (int j = 0; j < K; ++j) st[i * kN + j] = isfinite(S[i][j]) && isfinite(other[i][j]) ? other[i][j] : S[i][j];
}

// grid (units, 64 LG / (32 NCW RPT)); NCW warps compute (a warp: 32 / LG groups of LG lanes, RPT rows each), NSW warps stage
template <typename E, int LG, int NCW, int RPT, int NSW>
__global__ void __launch_bounds__(32 * (NCW + NSW)) wkv7_rows_kernel(int T, int H, float* __restrict__ state, const E* __restrict__ r_,
                                                        const E* __restrict__ w_, const E* __restrict__ k_, const E* __restrict__ v_,
                                                        const E* __restrict__ a_, const E* __restrict__ b_, E* __restrict__ y_) {
    extern __shared__ __align__(16) unsigned char smem_rows[];
    constexpr int kCh = NSW * kQ, NTH = 32 * (NCW + NSW);   // tokens staged at a time
    Staged<NSW>* buf = reinterpret_cast<Staged<NSW>*>(smem_rows);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int unit = blockIdx.x, C = H * kN;
    const i64 base = (i64)(unit / H) * T * C + (unit % H) * kN;
    const int nch = (T + kCh - 1) / kCh;

    if (warp >= NCW) {
        // ---- staging: a step of every chunk per warp, two keys per lane (those of the places 2 lane, 2 lane + 1 of a staged row) ----
        // (in registers one chunk ahead of the stores, asked for in L2 64 tokens ahead)
        const int q = warp - NCW, key = lane < 16 ? 8 * (lane >> 1) + 2 * (lane & 1) : 8 * ((lane - 16) >> 1) + 4 + 2 * (lane & 1);
        const E* src[6] = {w_, a_, b_, k_, r_, v_};
        const i64 o0 = base + (i64)q * kQ * C;
        Pair2<E> raw[6][kQ];
        auto fetch = [&](int c) {
            const int t = c * kCh + q * kQ;
            const i64 o = o0 + (i64)c * kCh * C + key;
#pragma unroll
            for (int x = 0; x < 6; ++x)
#pragma unroll
                for (int i = 0; i < kQ; ++i) raw[x][i] = load2(src[x] + o + (i64)i * C, t + i < T);
            if (lane < 24 && t + 64 + (lane & 3) < T) {   // one row per lane: 128 or 256 bytes
                const E* p = lane < 4 ? w_ : lane < 8 ? a_ : lane < 12 ? b_ : lane < 16 ? k_ : lane < 20 ? r_ : v_;
                p += o0 + (i64)(c * kCh + 64 + (lane & 3)) * C;
                prefetch_l2(p);
                if (sizeof(E) == 4) prefetch_l2(p + 32);
            }
        };
        const int yt = lane >= 24 ? 3 : lane >= 18 ? 2 : lane >= 14 ? 1 : 0, slot = lane < 12 ? lane : 12 + 8 * yt + lane - (yt == 3 ? 24 : yt == 2 ? 18 : yt == 1 ? 14 : 12);
        float odd = 0.f;
        fetch(0);
        for (int c = 0; c < nch; ++c) {
            const int t0 = c * kCh + q * kQ;
            float2 d[kQ], a[kQ], b[kQ], k[kQ], r[kQ], v[kQ];
#pragma unroll
            for (int i = 0; i < kQ; ++i) {
                const float2 w = decode2(raw[0][i]);
                d[i] = t0 + i < T ? make_float2(decay7(w.x), decay7(w.y)) : make_float2(1.f, 1.f);
                a[i] = decode2(raw[1][i]); b[i] = decode2(raw[2][i]); k[i] = decode2(raw[3][i]); r[i] = decode2(raw[4][i]); v[i] = decode2(raw[5][i]);
            }
            if (c + 1 < nch) fetch(c + 1);
            // every pair of tokens: b_s, k_s times the decays between s and t, against a_t (without token t's) and r_t (with it)
            float u[32];
#pragma unroll
            for (int s = 0; s < kQ; ++s) {
                float2 p = b[s], z = k[s];
                constexpr int first[kQ] = {12, 14, 18, 24};
                u[first[s] + 2 * s] = dot2(p, r[s]);
                u[first[s] + 2 * s + 1] = dot2(z, r[s]);
#pragma unroll
                for (int t = s + 1; t < kQ; ++t) {
                    u[(t - 1) * t + 2 * s] = dot2(p, a[t]);
                    u[(t - 1) * t + 2 * s + 1] = dot2(z, a[t]);
                    p = times(p, d[t]);
                    z = times(z, d[t]);
                    u[first[t] + 2 * s] = dot2(p, r[t]);
                    u[first[t] + 2 * s + 1] = dot2(z, r[t]);
                }
            }
            // the vectors of the step, with the decays of the tokens before them (a, r) and behind them (b, k): products of decays as
            // sums of two numbers, so that a vector is rounded once
            Exact2 w{d[0], make_float2(0.f, 0.f)}, e{d[kQ - 1], make_float2(0.f, 0.f)};
            r[0] = times(r[0], d[0]);
#pragma unroll
            for (int t = 1; t < kQ; ++t) {
                a[t] = times(a[t], w);
                w = times(w, d[t]);
                r[t] = times(r[t], w);
            }
#pragma unroll
            for (int s = kQ - 2; s >= 0; --s) {
                b[s] = times(b[s], e);
                k[s] = times(k[s], e);
                if (s > 0) e = times(e, d[s]);
            }
#pragma unroll
            for (int m = 16; m >= 1; m >>= 1) {   // sums over the lanes: lane x ends with u[x]
                const bool up = (lane & m) != 0;
#pragma unroll
                for (int i = 0; i < m; ++i) {
                    const float send = up ? u[i] : u[i + m], keep = up ? u[i + m] : u[i];
                    u[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
                }
            }
            if (c >= 2) bar_sync<3, NTH>(c & 1);   // the compute warps are done with the chunk before last
            Step& st = buf[c & 1].s[q];
#pragma unroll
            for (int i = 0; i < kQ; ++i) {
                *reinterpret_cast<float2*>(st.a[i] + 2 * lane) = a[i];
                *reinterpret_cast<float2*>(st.r[i] + 2 * lane) = r[i];
                *reinterpret_cast<float2*>(st.b[i] + 2 * lane) = b[i];
                *reinterpret_cast<float2*>(st.k[i] + 2 * lane) = k[i];
                *reinterpret_cast<float2*>(st.v[i] + key) = v[i];
            }
            *reinterpret_cast<float2*>(st.w + 2 * lane) = make_float2(w.hi.x + w.lo.x, w.hi.y + w.lo.y);
            st.u[slot] = u[0];
            check(odd, u[0]);   // every r is in one of these sums; all other values reach the state
            if (c + 1 == nch) st.odd = __any_sync(0xffffffffu, odd != 0.f);
            bar_arrive<1, NTH>(c & 1);
        }
        return;
    }

    // ---- the recurrence: RPT rows per group of LG lanes, four tokens per step -------------------------------------------------------
    constexpr int GPW = 32 / LG, KP = 32 / LG, TS = LG / 8;   // groups of a warp; pairs of keys of a lane; lanes per sum
    const int x = lane & (LG - 1), row0 = ((blockIdx.y * NCW + warp) * GPW + lane / LG) * RPT;
    float* st = state + (i64)unit * kN * kN + row0 * kN + first_key<LG>(x);
    f2 S[RPT][KP];
#pragma unroll
    for (int i = 0; i < RPT; ++i)
#pragma unroll
        for (int h = 0; h < KP / 2; ++h) {
            const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(st + i * kN + 4 * h);
            S[i][2 * h] = p.x; S[i][2 * h + 1] = p.y;
        }
    for (int c = 0; c < nch; ++c) {
        bar_sync<1, NTH>(c & 1);
#pragma unroll 1
        for (int q = 0; q < kCh / kQ; ++q) {
            const Step& s = buf[c & 1].s[q];
            float p[RPT][8];   // S.r~_t, S.a~_t: parts of this lane
#pragma unroll
            for (int t = 0; t < kQ; ++t) {
                const Keys<LG> a = load_keys<LG>(s.a[t], x), r = load_keys<LG>(s.r[t], x);
#pragma unroll
                for (int i = 0; i < RPT; ++i) { p[i][4 + t] = dot_keys<LG>(S[i], a); p[i][t] = dot_keys<LG>(S[i], r); }
            }
            float own[RPT];
#pragma unroll
            for (int i = 0; i < RPT; ++i) own[i] = reduce8_over<LG>(p[i], x);
            // while these are under way: S <- S w + sum v_s k^_s
            float v[kQ][RPT];
            {
                const Keys<LG> w = load_keys<LG>(s.w, x);
#pragma unroll
                for (int i = 0; i < RPT; ++i)
#pragma unroll
                    for (int e = 0; e < KP; ++e) S[i][e] = mul2(S[i][e], w.x[e]);
            }
#pragma unroll
            for (int t = 0; t < kQ; ++t) {
                const Keys<LG> k = load_keys<LG>(s.k[t], x);
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    v[t][i] = s.v[t][row0 + i];
                    const f2 vv = pack2(v[t][i], v[t][i]);
#pragma unroll
                    for (int e = 0; e < KP; ++e) S[i][e] = fma2(k.x[e], vv, S[i][e]);
                }
            }
            float u[12], g[8];
#pragma unroll
            for (int i = 0; i < 3; ++i) *reinterpret_cast<float4*>(u + 4 * i) = *reinterpret_cast<const float4*>(s.u + 4 * i);
            const int ty = (x / TS) & 3;   // the token whose y this lane makes (lanes with an S.a~ repeat one)
#pragma unroll
            for (int i = 0; i < 2; ++i) *reinterpret_cast<float4*>(g + 4 * i) = *reinterpret_cast<const float4*>(s.u + 12 + 8 * ty + 4 * i);
            float sa[kQ][RPT];
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                float z[kQ];
#pragma unroll
                for (int t = 0; t < kQ; ++t) z[t] = __shfl_sync(0xffffffffu, own[i], (4 + t) * TS, LG);
#pragma unroll
                for (int t = 0; t < kQ; ++t) {
#pragma unroll
                    for (int e = 0; e < t; ++e) z[t] = fmaf(v[e][i], u[(t - 1) * t + 2 * e + 1], z[t]);
#pragma unroll
                    for (int e = 0; e < t; ++e) z[t] = fmaf(sa[e][i], u[(t - 1) * t + 2 * e], z[t]);
                    sa[t][i] = z[t];
                }
            }
            // sum sa_s b^_s by itself, then onto the state (one rounding at the size of the state, not four)
            f2 sb[RPT][KP];
#pragma unroll
            for (int t = 0; t < kQ; ++t) {
                const Keys<LG> b = load_keys<LG>(s.b[t], x);
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    const f2 sv = pack2(sa[t][i], sa[t][i]);
#pragma unroll
                    for (int e = 0; e < KP; ++e) sb[i][e] = t ? fma2(b.x[e], sv, sb[i][e]) : mul2(b.x[e], sv);
                }
            }
#pragma unroll
            for (int i = 0; i < RPT; ++i)
#pragma unroll
                for (int e = 0; e < KP; ++e) S[i][e] = add2(S[i][e], sb[i][e]);
            float y[RPT];
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                y[i] = own[i];
#pragma unroll
                for (int e = 0; e < kQ; ++e)
                    if (e <= ty) y[i] = fmaf(sa[e][i], g[2 * e], fmaf(v[e][i], g[2 * e + 1], y[i]));   // (g is not set for later tokens)
            }
            const int t = c * kCh + kQ * q + ty;
            if (x < 4 * TS && x % TS == 0 && t < T) store_rows<E, RPT>(y_ + base + (i64)t * C + row0, y);
        }
        if (c + 2 < nch) bar_arrive<3, NTH>(c & 1);
    }
    float bad = 0.f;
#pragma unroll
    for (int i = 0; i < RPT; ++i)
#pragma unroll
        for (int e = 0; e < KP; ++e) check(bad, sum2(S[i][e]));
    for (int q = 0; q < NSW; ++q)
        if (buf[(nch - 1) & 1].s[q].odd) bad = 1.f;
    if (__any_sync(0xffffffffu, bad != 0.f)) {   // (an infinity never leaves a state: d > 0.5; r does not enter it)
        float other[RPT][2 * KP];
#pragma unroll
        for (int i = 0; i < RPT; ++i)
#pragma unroll
            for (int e = 0; e < KP; ++e) unpack2(S[i][e], other[i][2 * e], other[i][2 * e + 1]);
        __syncwarp();   // (other lanes of the warp have written the y that it looks at)
        rows_again<E, LG, RPT>(T, C, base, row0, x, st, r_, w_, k_, v_, a_, b_, y_, other);
        return;
    }
#pragma unroll
    for (int i = 0; i < RPT; ++i)
#pragma unroll
        for (int h = 0; h < KP / 2; ++h) *reinterpret_cast<ulonglong2*>(st + i * kN + 4 * h) = make_ulonglong2(S[i][2 * h], S[i][2 * h + 1]);
}

template <typename E, int LG, int NCW, int RPT, int NSW>
int launch_rows(int B, int T, int H, float* state, const void* r, const void* w, const void* k, const void* v, const void* a,
                const void* b, void* y, cudaStream_t st) {
    constexpr int smem = 2 * sizeof(Staged<NSW>);
    const cudaError_t e = allow_smem<wkv7_rows_kernel<E, LG, NCW, RPT, NSW>>(smem);
    RWKV_REQUIRE(e == cudaSuccess, RWKVB200_ECUDA, "wkv7_state_update: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    wkv7_rows_kernel<E, LG, NCW, RPT, NSW><<<dim3(B * H, kN * LG / (32 * NCW * RPT)), 32 * (NCW + NSW), smem, st>>>(
        T, H, state, (const E*)r, (const E*)w, (const E*)k, (const E*)v, (const E*)a, (const E*)b, (E*)y);
    return check_launch("wkv7_state_update(rows)");
}

template <typename E>
int update(int B, int T, int H, float* state, const void* r, const void* w, const void* k, const void* v, const void* a, const void* b,
           void* y, int sms, cudaStream_t st) {
    if (T == 1) {
        wkv7_decode_kernel<E><<<B * H, 128, 0, st>>>(state, (const E*)r, (const E*)w, (const E*)k, (const E*)v, (const E*)a, (const E*)b, (E*)y);
        return check_launch("wkv7_state_update(decode)");
    }
    // The fewest rows per block that still give every block an SM of its own (blocks that share one share its shared-memory
    // bandwidth: with a token as a step 64 units took 356 us in blocks of 16 rows and 284 us in blocks of 32); with more units than
    // SMs / 2 the most rows per thread, which read every staged vector for four rows.
    const int units = B * H;
    if (units * 4 <= sms) return launch_rows<E, 16, 4, 2, 8>(B, T, H, state, r, w, k, v, a, b, y, st);
    if (units * 2 <= sms) return launch_rows<E, 8, 4, 2, 4>(B, T, H, state, r, w, k, v, a, b, y, st);
    return launch_rows<E, 8, 4, 4, 4>(B, T, H, state, r, w, k, v, a, b, y, st);
}

}  // namespace

int wkv7_update64(int dtype, int B, int T, int H, float* state, const void* r, const void* w, const void* k, const void* v,
                  const void* a, const void* b, void* y, int sms, cudaStream_t st) {
    return dtype == RWKVB200_F32 ? update<float>(B, T, H, state, r, w, k, v, a, b, y, sms, st)
                                 : update<bf16>(B, T, H, state, r, w, k, v, a, b, y, sms, st);
}

}  // namespace rwkvb200
