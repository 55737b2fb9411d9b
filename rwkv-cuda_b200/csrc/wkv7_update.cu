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
// chain from one token's sa to the next (a dot product over 64 keys and its reduction over lanes) and, with many rows on
// an SM, the shared-memory reads of the token's vectors (2 / RPT wavefronts per row and vector whatever the lane split).
// Against the chain: 8 or 16 lanes own a row, and the dot product runs one token ahead of sa: with
// G_t = S_{t-1} d_t + v_t k_t (no sa_t in it) and beta_t = b_t.a_{t+1} (one scalar per token),
//     sa_{t+1} = G_t.a_{t+1} + sa_t beta_t          S_t = G_t + sa_t b_t
// so the reduction of token t+1 overlaps the update of token t.  Against the reads: RPT rows per thread.
// NCW warps compute, four stage the next 16 tokens in shared memory (fp32: d, b, k, r, v of token t and a of token t+1)
// behind named barriers.  Multiply-adds are packed in pairs (fma.rn.f32x2), y is reduced for eight tokens at a time.
// One sequence of 1999 tokens, 32 heads: 2010 us for the general-shape kernel, 212 us here (106 ns per token); 256 units
// 2045 -> 870 us.
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
__device__ __forceinline__ int staged_at(int ch) { return ((ch & 4) << 3) + ((ch >> 3) << 2) + (ch & 3); }
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
template <int LG>
__device__ __forceinline__ float row_sum(float x) {
#pragma unroll
    for (int m = 1; m < LG; m <<= 1) x += __shfl_xor_sync(0xffffffffu, x, m);
    return x;
}

constexpr int kCh = 16;                              // tokens staged at a time
struct __align__(16) Token { float d[kN], b[kN], k[kN], r[kN], an[kN], v[kN]; };
struct __align__(16) Staged { Token t[kCh]; float beta[kCh]; };
constexpr int kRowsSmem = 2 * sizeof(Staged);

// 8 consecutive elements as loaded, and decoded
template <typename E>
struct Raw8 { uint4 q[sizeof(E) / 2]; };
template <typename E>
__device__ __forceinline__ Raw8<E> load8(const E* p, bool in) {
    Raw8<E> x;
#pragma unroll
    for (int i = 0; i < (int)sizeof(E) / 2; ++i) x.q[i] = in ? __ldg(reinterpret_cast<const uint4*>(p) + i) : make_uint4(0u, 0u, 0u, 0u);
    return x;
}
__device__ __forceinline__ void decode8(const Raw8<float>& p, float (&x)[8]) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        x[4 * i] = __uint_as_float(p.q[i].x); x[4 * i + 1] = __uint_as_float(p.q[i].y);
        x[4 * i + 2] = __uint_as_float(p.q[i].z); x[4 * i + 3] = __uint_as_float(p.q[i].w);
    }
}
__device__ __forceinline__ void decode8(const Raw8<bf16>& p, float (&x)[8]) {
    const uint32_t u[4] = {p.q[0].x, p.q[0].y, p.q[0].z, p.q[0].w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { x[2 * i] = __uint_as_float(u[i] << 16); x[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u); }
}
__device__ __forceinline__ void prefetch_l2(const void* p) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(__cvta_generic_to_global(p)));
}
__device__ __forceinline__ void store8(float* row, int l8, const float (&x)[8]) {
    *reinterpret_cast<float4*>(row + 4 * l8) = make_float4(x[0], x[1], x[2], x[3]);
    *reinterpret_cast<float4*>(row + 32 + 4 * l8) = make_float4(x[4], x[5], x[6], x[7]);
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

// grid (units, 64 / (16 RPT)); 4 compute warps (a warp: 4 groups of 8 lanes, RPT rows each) and 4 staging warps
template <typename E, int LG, int NCW, int RPT>
__global__ void __launch_bounds__(32 * (NCW + 4)) wkv7_rows_kernel(int T, int H, float* __restrict__ state, const E* __restrict__ r_,
                                                        const E* __restrict__ w_, const E* __restrict__ k_, const E* __restrict__ v_,
                                                        const E* __restrict__ a_, const E* __restrict__ b_, E* __restrict__ y_) {
    extern __shared__ __align__(16) unsigned char smem_rows[];
    Staged* buf = reinterpret_cast<Staged*>(smem_rows);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l8 = lane & 7;
    const int unit = blockIdx.x, C = H * kN;
    const i64 base = (i64)(unit / H) * T * C + (unit % H) * kN;
    const int nch = (T + kCh - 1) / kCh;
    constexpr int NTH = 32 * (NCW + 4);

    if (warp >= NCW) {
        // ---- staging: this lane has keys 8 l8 .. of token 4 (warp - NCW) + lane / 8 of every chunk --------------
        // (in registers one chunk ahead of the stores, asked for in L2 four chunks ahead)
        const int q = 4 * (warp - NCW) + (lane >> 3);
        const E* src[6] = {w_, b_, k_, r_, v_, a_ + C};   // a: of the token after
        const i64 o0 = base + (i64)q * C + 8 * l8;
        Raw8<E> raw[6];
        auto fetch = [&](int c) {
            const int t = c * kCh + q;
            const i64 o = o0 + (i64)c * kCh * C;
#pragma unroll
            for (int x = 0; x < 6; ++x) raw[x] = load8(src[x] + o, t + (x == 5) < T);
            if (t + 4 * kCh + 1 < T && (l8 & (64 / sizeof(E) / 8 * 2 - 1)) == 0)   // one lane per 128-byte line
#pragma unroll
                for (int x = 0; x < 6; ++x) prefetch_l2(src[x] + o + (i64)4 * kCh * C);
        };
        fetch(0);
        for (int c = 0; c < nch; ++c) {
            const bool in = c * kCh + q < T;
            float w[8], b[8], k[8], r[8], v[8], an[8];
            decode8(raw[0], w); decode8(raw[1], b); decode8(raw[2], k); decode8(raw[3], r); decode8(raw[4], v); decode8(raw[5], an);
            if (c + 1 < nch) fetch(c + 1);
            float beta = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) { w[i] = in ? decay7(w[i]) : 1.f; beta = fmaf(b[i], an[i], beta); }
#pragma unroll
            for (int m = 1; m < 8; m <<= 1) beta += __shfl_xor_sync(0xffffffffu, beta, m);
            if (c >= 2) bar_sync<3, NTH>(c & 1);   // the compute warps are done with the chunk before last
            Staged& s = buf[c & 1];
            Token& d = s.t[q];
            store8(d.d, l8, w); store8(d.b, l8, b); store8(d.k, l8, k);
            store8(d.r, l8, r); store8(d.an, l8, an); store8(d.v, l8, v);
            if (l8 == 0) s.beta[q] = beta;
            bar_arrive<1, NTH>(c & 1);
        }
        return;
    }

    // ---- the recurrence: RPT rows per group of LG lanes -----------------------------------------------------------
    constexpr int GPW = 32 / LG, KP = 32 / LG;   // groups of a warp; pairs of keys of a lane
    const int x = lane & (LG - 1), row0 = ((blockIdx.y * NCW + warp) * GPW + lane / LG) * RPT;
    float* st = state + (i64)unit * kN * kN + row0 * kN + first_key<LG>(x);
    f2 S[RPT][KP];
    float sa[RPT];
    {
        Keys<LG> a;
#pragma unroll
        for (int h = 0; h < KP / 2; ++h) {
            const float4 q = load4(a_ + base + first_key<LG>(x) + 4 * h);
            a.x[2 * h] = pack2(q.x, q.y); a.x[2 * h + 1] = pack2(q.z, q.w);
        }
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
#pragma unroll
            for (int h = 0; h < KP / 2; ++h) {
                const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(st + i * kN + 4 * h);
                S[i][2 * h] = p.x; S[i][2 * h + 1] = p.y;
            }
            sa[i] = row_sum<LG>(dot_keys<LG>(S[i], a));
        }
    }
    for (int c = 0; c < nch; ++c) {
        bar_sync<1, NTH>(c & 1);
        const Staged& s = buf[c & 1];
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
            float yp[RPT][8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const Token& tk = s.t[8 * half + q];
                const float beta = s.beta[8 * half + q];
                const Keys<LG> d = load_keys<LG>(tk.d, x), k = load_keys<LG>(tk.k, x), an = load_keys<LG>(tk.an, x), b = load_keys<LG>(tk.b, x),
                               r = load_keys<LG>(tk.r, x);
                float z[RPT];
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    const float v = tk.v[staged_at(row0 + i)];
                    const f2 vv = pack2(v, v);
#pragma unroll
                    for (int e = 0; e < KP; ++e) S[i][e] = fma2(S[i][e], d.x[e], mul2(k.x[e], vv));   // G_t
                    z[i] = dot_keys<LG>(S[i], an);
                }
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    const f2 sv = pack2(sa[i], sa[i]);
#pragma unroll
                    for (int e = 0; e < KP; ++e) S[i][e] = fma2(sv, b.x[e], S[i][e]);                 // S_t
                    yp[i][q] = dot_keys<LG>(S[i], r);
                    sa[i] = fmaf(sa[i], beta, row_sum<LG>(z[i]));                                     // sa_{t+1}
                }
            }
            // sums over the lanes of a row for 8 tokens: every lane of a row ends with one token (pairs of lanes when LG = 16)
            constexpr int TS = LG / 8;
            const int t = c * kCh + 8 * half + x / TS;
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
#pragma unroll
                for (int m = 4; m >= 1; m >>= 1) {
                    const bool up = (x & (m * TS)) != 0;
#pragma unroll
                    for (int e = 0; e < m; ++e) {
                        const float send = up ? yp[i][e] : yp[i][e + m], keep = up ? yp[i][e + m] : yp[i][e];
                        yp[i][e] = keep + __shfl_xor_sync(0xffffffffu, send, m * TS);
                    }
                }
                if (LG == 16) yp[i][0] += __shfl_xor_sync(0xffffffffu, yp[i][0], 1);
                if (t < T && x % TS == 0) y_[base + (i64)t * C + row0 + i] = from_f<E>(yp[i][0]);
            }
        }
        if (c + 2 < nch) bar_arrive<3, NTH>(c & 1);
    }
#pragma unroll
    for (int i = 0; i < RPT; ++i)
#pragma unroll
        for (int h = 0; h < KP / 2; ++h) *reinterpret_cast<ulonglong2*>(st + i * kN + 4 * h) = make_ulonglong2(S[i][2 * h], S[i][2 * h + 1]);
}

template <typename E, int LG, int NCW, int RPT>
int launch_rows(int B, int T, int H, float* state, const void* r, const void* w, const void* k, const void* v, const void* a,
                const void* b, void* y, cudaStream_t st) {
    const cudaError_t e = allow_smem<wkv7_rows_kernel<E, LG, NCW, RPT>>(kRowsSmem);
    RWKV_REQUIRE(e == cudaSuccess, RWKVB200_ECUDA, "wkv7_state_update: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    wkv7_rows_kernel<E, LG, NCW, RPT><<<dim3(B * H, kN * LG / (32 * NCW * RPT)), 32 * (NCW + 4), kRowsSmem, st>>>(
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
    // bandwidth: 64 units in blocks of 16 rows take 356 us, in blocks of 32 rows 284 us); with more units than SMs / 2 the
    // most rows per thread, which read every staged vector for four rows (T = 1999: 128 units 480 us, 256 units 870 us).
    const int units = B * H;
    if (units * 4 <= sms) return launch_rows<E, 16, 4, 2>(B, T, H, state, r, w, k, v, a, b, y, st);
    if (units * 2 <= sms) return launch_rows<E, 8, 4, 2>(B, T, H, state, r, w, k, v, a, b, y, st);
    return launch_rows<E, 8, 4, 4>(B, T, H, state, r, w, k, v, a, b, y, st);
}

}  // namespace

int wkv7_update64(int dtype, int B, int T, int H, float* state, const void* r, const void* w, const void* k, const void* v,
                  const void* a, const void* b, void* y, int sms, cudaStream_t st) {
    return dtype == RWKVB200_F32 ? update<float>(B, T, H, state, r, w, k, v, a, b, y, sms, st)
                                 : update<bf16>(B, T, H, state, r, w, k, v, a, b, y, sms, st);
}

}  // namespace rwkvb200
