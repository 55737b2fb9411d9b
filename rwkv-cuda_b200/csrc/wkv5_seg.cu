// RWKV-5 training in fp32 arithmetic (fp32 activations; bf16 where the tensor-core kernels do not apply), any head size
// N <= 128, split over time.
//
// Per (batch, head), S indexed [key j][value i], w the decay of a key:
//   y_t[i] = sum_j r_t[j] S_{t-1}[j,i] + v_t[i] sum_j r_t u k_t      S_t[j,i] = w[j] S_{t-1}[j,i] + k_t[j] v_t[i]
// wkv5.cu walks T tokens with one thread per state line: 0.4 to 0.9 us per token and sweep, with 8 to 128 units for 148 SMs.
// The state is linear in its start, so T is cut into segments of kSeg tokens which are all worked on at the same time:
//   local   the end state of every segment from a zero start: sum_s w^{n-1-s} k_s v_s^T, one multiply-add per state element
//           and token because the powers of w are put on k when it is staged (they are <= 1: nothing can overflow, whatever w is);
//   scan    start states of the segments, in place: S <- S diag(w^n) + local;
//   y       every segment again, token by token from its start state.
// Backward: the same two steps for the adjoint D = dL/dS (k, v -> r, gy, time reversed), then one block per segment whose three
// groups of threads walk it at the same time: S forward (gr), D by key lines backward (gk), D by value lines backward (gv).
// The decays of a segment act on its own outputs and on its end state: with Z = dS/dlog w counted from the segment's start
// (Z_0 = 0, Z <- w (Z + S)), the segment's part of dL/dlog w is sum_t r_t sum_i gy_t Z_t + sum_i D_end Z_end.  (The sum over
// states and gradients that needs no Z cancels for fast decays: 10 % error in gw at w = exp(-exp(3)).)
// Inputs are staged in shared memory once per segment, so the token loops have no barrier; multiply-adds are packed in pairs.
// fp32, B8 T512 H16 N64, forward + backward on a B200: 1285 us with wkv5.cu, 635 us here.
#include "wkv5_seg.cuh"
#include "packed.cuh"

namespace rwkvb200 {
namespace {

constexpr int kSeg = kWkv5Seg;

// Stages `n` tokens of a (T, C) tensor into dst[kSeg][NMAX] as fp32, zero where there is no token or channel.
template <typename E, int NMAX>
__device__ __forceinline__ void stage(float* dst, const E* __restrict__ src, int n, int C, int N, int tid, int nth) {
    for (int x = tid; x < kSeg * NMAX; x += nth) {
        const int t = x / NMAX, j = x % NMAX;
        dst[x] = (t < n && j < N) ? to_f(src[(i64)t * C + j]) : 0.f;
    }
}
template <typename E>
__device__ __forceinline__ float log_decay(const E* w_raw) { return -expf(to_f(*w_raw)); }   // log w = -exp(w_raw)
__device__ __forceinline__ float power(float lw, int e) { return e == 0 ? 1.f : expf(lw * (float)e); }   // w^e, also for w = 0

// state line of a thread: element e at p[e * stride]
template <int NMAX>
__device__ __forceinline__ void load_line(f2 (&s)[NMAX / 2], const float* p, int stride, int N, bool live) {
#pragma unroll
    for (int e = 0; e < NMAX / 2; ++e)
        s[e] = pack2(live && 2 * e < N ? p[(i64)(2 * e) * stride] : 0.f, live && 2 * e + 1 < N ? p[(i64)(2 * e + 1) * stride] : 0.f);
}
template <int NMAX>
__device__ __forceinline__ void store_line(const f2 (&s)[NMAX / 2], float* p, int stride, int N, bool live) {
#pragma unroll
    for (int e = 0; e < NMAX / 2; ++e) {
        float lo, hi;
        unpack2(s[e], lo, hi);
        if (live && 2 * e < N) p[(i64)(2 * e) * stride] = lo;
        if (live && 2 * e + 1 < N) p[(i64)(2 * e + 1) * stride] = hi;
    }
}

// grid (segments, units), NMAX threads, thread = value i.  REV = false: a = k, b = v; REV = true: a = r, b = gy.
template <typename E, int NMAX, bool REV>
__global__ void __launch_bounds__(NMAX, NMAX == 128 ? 2 : 512 / NMAX) seg_local_kernel(int T, int C, int H, int N, const E* __restrict__ a_, const E* __restrict__ b_,
                                                         const E* __restrict__ w_, float* __restrict__ states) {
    __shared__ __align__(16) float as[kSeg * NMAX];
    const int seg = blockIdx.x, unit = blockIdx.y, h = unit % H, i = threadIdx.x;
    const int n = min(kSeg, T - seg * kSeg);
    const i64 base = ((i64)(unit / H) * T + seg * kSeg) * C + h * N;
    const bool live = i < N;
    {   // a, times the decay between its token and the end (REV: the start) of the segment; thread = key here
        const float lw = live ? log_decay(w_ + h * N + i) : 0.f;
        for (int t = 0; t < kSeg; ++t)
            as[t * NMAX + i] = (live && t < n) ? to_f(a_[base + (i64)t * C + i]) * power(lw, REV ? t : n - 1 - t) : 0.f;
    }
    __syncthreads();
    f2 s[NMAX / 2];
#pragma unroll
    for (int e = 0; e < NMAX / 2; ++e) s[e] = 0ull;
#pragma unroll 2
    for (int t = 0; t < n; ++t) {
        const float b = live ? to_f(b_[base + (i64)t * C + i]) : 0.f;
        const f2 bb = pack2(b, b);
        const ulonglong2* ap = reinterpret_cast<const ulonglong2*>(as + t * NMAX);
#pragma unroll
        for (int e = 0; e < NMAX / 4; ++e) {
            const ulonglong2 q = ap[e];
            s[2 * e] = fma2(q.x, bb, s[2 * e]);
            s[2 * e + 1] = fma2(q.y, bb, s[2 * e + 1]);
        }
    }
    store_line<NMAX>(s, states + ((i64)unit * gridDim.x + seg) * N * N + i, N, N, live);
}

// In place: local end states -> state before each segment (REV: adjoint after each segment).  One thread per state element.
template <typename E, bool REV>
__global__ void __launch_bounds__(256) seg_scan_kernel(int T, int H, int N, int nseg, const E* __restrict__ w_, float* __restrict__ states) {
    const int e = blockIdx.x * 256 + threadIdx.x, unit = blockIdx.y;
    if (e >= N * N) return;
    const float lw = log_decay(w_ + (unit % H) * N + e / N);
    const float full = expf(lw * kSeg), tail = expf(lw * (float)(T - (nseg - 1) * kSeg));
    float* p = states + (i64)unit * nseg * N * N + e;
    constexpr int AHEAD = 8;
    float cur = 0.f;
    for (int k0 = 0; k0 < nseg; k0 += AHEAD) {   // the loads of AHEAD segments are in flight together
        float x[AHEAD];
#pragma unroll
        for (int q = 0; q < AHEAD; ++q)
            if (k0 + q < nseg) x[q] = p[(i64)(REV ? nseg - 1 - k0 - q : k0 + q) * N * N];
#pragma unroll
        for (int q = 0; q < AHEAD; ++q)
            if (k0 + q < nseg) {
                const int k = REV ? nseg - 1 - k0 - q : k0 + q;
                p[(i64)k * N * N] = cur;
                cur = fmaf(cur, k == nseg - 1 ? tail : full, x[q]);
            }
    }
}

// grid (segments, units), NMAX threads, thread = value i
template <typename E, int NMAX>
__global__ void __launch_bounds__(NMAX, NMAX == 128 ? 2 : 512 / NMAX) seg_y_kernel(int T, int C, int H, int N, const E* __restrict__ r_, const E* __restrict__ k_,
                                                     const E* __restrict__ v_, const E* __restrict__ w_, const E* __restrict__ u_,
                                                     const float* __restrict__ states, E* __restrict__ y_) {
    __shared__ __align__(16) float rs[kSeg * NMAX], ks[kSeg * NMAX], ws[NMAX], us[NMAX], ruk[kSeg];
    const int seg = blockIdx.x, unit = blockIdx.y, h = unit % H, i = threadIdx.x;
    const int n = min(kSeg, T - seg * kSeg);
    const i64 base = ((i64)(unit / H) * T + seg * kSeg) * C + h * N;
    const bool live = i < N;
    stage<E, NMAX>(rs, r_ + base, n, C, N, i, NMAX);
    stage<E, NMAX>(ks, k_ + base, n, C, N, i, NMAX);
    ws[i] = live ? expf(log_decay(w_ + h * N + i)) : 0.f;
    us[i] = live ? to_f(u_[h * N + i]) : 0.f;
    f2 s[NMAX / 2];
    load_line<NMAX>(s, states + ((i64)unit * gridDim.x + seg) * N * N + i, N, N, live);
    __syncthreads();
    for (int t = i / 32; t < n; t += NMAX / 32) {   // the bonus of a token: one warp each
        float x = 0.f;
        for (int j = i & 31; j < NMAX; j += 32) x = fmaf(rs[t * NMAX + j] * us[j], ks[t * NMAX + j], x);
#pragma unroll
        for (int m = 16; m; m >>= 1) x += __shfl_xor_sync(0xffffffffu, x, m);
        if ((i & 31) == 0) ruk[t] = x;
    }
    __syncthreads();
    float vn = live ? to_f(v_[base + i]) : 0.f;
    for (int t = 0; t < n; ++t) {
        const float v = vn;
        if (t + 1 < n && live) vn = to_f(v_[base + (i64)(t + 1) * C + i]);
        const f2 vv = pack2(v, v);
        f2 y0 = 0ull, y1 = 0ull;
        const ulonglong2 *rp = reinterpret_cast<const ulonglong2*>(rs + t * NMAX), *kp = reinterpret_cast<const ulonglong2*>(ks + t * NMAX),
                         *wp = reinterpret_cast<const ulonglong2*>(ws);
#pragma unroll
        for (int e = 0; e < NMAX / 4; ++e) {
            const ulonglong2 r = rp[e], k = kp[e], w = wp[e];
            y0 = fma2(r.x, s[2 * e], y0);
            y1 = fma2(r.y, s[2 * e + 1], y1);
            s[2 * e] = fma2(s[2 * e], w.x, mul2(k.x, vv));
            s[2 * e + 1] = fma2(s[2 * e + 1], w.y, mul2(k.y, vv));
        }
        if (live) y_[base + (i64)t * C + i] = from_f<E>(fmaf(v, ruk[t], sum2(y0) + sum2(y1)));
    }
}

// grid (segments, units), 4 NMAX threads: the first half = key lines of S and Z, two neighbouring threads per line; then NMAX
// threads for the key lines of D and NMAX for its value lines
template <int NMAX>
struct BwdSmem {
    float r[kSeg * NMAX], k[kSeg * NMAX], v[kSeg * NMAX], g[kSeg * NMAX];
    float w[NMAX], u[NMAX], vg[kSeg], ruk[kSeg];
};

template <typename E, int NMAX>
__global__ void __launch_bounds__(4 * NMAX, NMAX == 128 ? 1 : 2) seg_backward_kernel(int T, int C, int H, int N, const E* __restrict__ r_, const E* __restrict__ k_,
                                                                const E* __restrict__ v_, const E* __restrict__ w_, const E* __restrict__ u_,
                                                                const E* __restrict__ gy_, const float* __restrict__ S_,
                                                                const float* __restrict__ D_, E* __restrict__ gr_, E* __restrict__ gk_,
                                                                E* __restrict__ gv_, float* __restrict__ partial_) {
    extern __shared__ __align__(16) unsigned char smem_seg[];
    BwdSmem<NMAX>& sm = *reinterpret_cast<BwdSmem<NMAX>*>(smem_seg);
    const int seg = blockIdx.x, unit = blockIdx.y, h = unit % H, grp = threadIdx.x / NMAX, half = threadIdx.x & 1;
    const int i = grp < 2 ? threadIdx.x >> 1 : threadIdx.x % NMAX;   // line
    constexpr int NTH = 4 * NMAX, HP = NMAX / 4;                      // pairs of half a line
    const int n = min(kSeg, T - seg * kSeg);
    const i64 base = ((i64)(unit / H) * T + seg * kSeg) * C + h * N;
    const bool live = i < N;
    const float* S0 = S_ + ((i64)unit * gridDim.x + seg) * N * N;
    const float* D0 = D_ + ((i64)unit * gridDim.x + seg) * N * N;
    stage<E, NMAX>(sm.r, r_ + base, n, C, N, threadIdx.x, NTH);
    stage<E, NMAX>(sm.k, k_ + base, n, C, N, threadIdx.x, NTH);
    stage<E, NMAX>(sm.v, v_ + base, n, C, N, threadIdx.x, NTH);
    stage<E, NMAX>(sm.g, gy_ + base, n, C, N, threadIdx.x, NTH);
    const float lw = live ? log_decay(w_ + h * N + i) : 0.f, w = live ? expf(lw) : 0.f, u = live ? to_f(u_[h * N + i]) : 0.f;
    if (grp == 2) { sm.w[i] = w; sm.u[i] = u; }
    f2 s[NMAX / 2];   // half of S[key i][:] and of Z[key i][:], D[key i][:] or D[:][value i]
    if (grp < 2) {
#pragma unroll
        for (int e = 0; e < HP; ++e) {   // (neighbouring float4s go to the two halves)
            const int j = 8 * (e >> 1) + 4 * half + 2 * (e & 1);
            s[e] = pack2(live && j < N ? S0[(i64)i * N + j] : 0.f, live && j + 1 < N ? S0[(i64)i * N + j + 1] : 0.f);
            s[HP + e] = 0ull;
        }
    } else if (grp == 2) load_line<NMAX>(s, D0 + (i64)i * N, 1, N, live);
    else load_line<NMAX>(s, D0 + i, N, N, live);
    __syncthreads();
    for (int t = threadIdx.x / 32; t < n; t += NTH / 32) {   // sums of a token over its channels: one warp each
        float x = 0.f, z = 0.f;
        for (int j = threadIdx.x & 31; j < NMAX; j += 32) {
            x = fmaf(sm.r[t * NMAX + j] * sm.u[j], sm.k[t * NMAX + j], x);
            z = fmaf(sm.v[t * NMAX + j], sm.g[t * NMAX + j], z);
        }
#pragma unroll
        for (int m = 16; m; m >>= 1) { x += __shfl_xor_sync(0xffffffffu, x, m); z += __shfl_xor_sync(0xffffffffu, z, m); }
        if ((threadIdx.x & 31) == 0) { sm.ruk[t] = x; sm.vg[t] = z; }
    }
    __syncthreads();
    const f2 ww = pack2(w, w);
    float gw = 0.f, gu = 0.f;
    if (grp < 2) {
        for (int t = 0; t < n; ++t) {
            const float r = sm.r[t * NMAX + i], k = sm.k[t * NMAX + i], vg = sm.vg[t];
            const f2 kk = pack2(k, k);
            const ulonglong2 *vp = reinterpret_cast<const ulonglong2*>(sm.v + t * NMAX) + half, *gp = reinterpret_cast<const ulonglong2*>(sm.g + t * NMAX) + half;
            f2 a0 = 0ull, a1 = 0ull, z0 = 0ull, z1 = 0ull;
#pragma unroll
            for (int e = 0; e < HP / 2; ++e) {
                const ulonglong2 v = vp[2 * e], g = gp[2 * e];
                f2 &s0 = s[2 * e], &s1 = s[2 * e + 1], &y0 = s[HP + 2 * e], &y1 = s[HP + 2 * e + 1];
                a0 = fma2(s0, g.x, a0);
                a1 = fma2(s1, g.y, a1);
                z0 = fma2(y0, g.x, z0);
                z1 = fma2(y1, g.y, z1);
                s0 = mul2(s0, ww);
                s1 = mul2(s1, ww);
                y0 = fma2(y0, ww, s0);
                y1 = fma2(y1, ww, s1);
                s0 = fma2(v.x, kk, s0);
                s1 = fma2(v.y, kk, s1);
            }
            float sg = sum2(a0) + sum2(a1);
            sg += __shfl_xor_sync(0xffffffffu, sg, 1);
            if (live && half == 0) gr_[base + (i64)t * C + i] = from_f<E>(fmaf(u * k, vg, sg));
            gw = fmaf(r, sum2(z0) + sum2(z1), gw);
            gu = fmaf(r * k, vg, gu);
        }
        f2 a0 = 0ull;   // sum over values of D_end Z_end
#pragma unroll
        for (int e = 0; e < HP; ++e) {
            const int j = 8 * (e >> 1) + 4 * half + 2 * (e & 1);
            a0 = fma2(pack2(live && j < N ? D0[(i64)i * N + j] : 0.f, live && j + 1 < N ? D0[(i64)i * N + j + 1] : 0.f), s[HP + e], a0);
        }
        gw += sum2(a0);
        gw += __shfl_xor_sync(0xffffffffu, gw, 1);
        if (live && half == 0) {
            float* p = partial_ + ((i64)(unit / H) * gridDim.x + seg) * 2 * C + h * N + i;
            p[0] = lw * gw;   // d log w / d w_raw = log w
            p[C] = gu;
        }
    } else if (grp == 2) {
        for (int t = n - 1; t >= 0; --t) {
            const float r = sm.r[t * NMAX + i];
            const f2 rr = pack2(r, r);
            const ulonglong2 *vp = reinterpret_cast<const ulonglong2*>(sm.v + t * NMAX), *gp = reinterpret_cast<const ulonglong2*>(sm.g + t * NMAX);
            f2 a0 = 0ull, a1 = 0ull;
#pragma unroll
            for (int e = 0; e < NMAX / 4; ++e) {
                const ulonglong2 v = vp[e], g = gp[e];
                a0 = fma2(s[2 * e], v.x, a0);
                a1 = fma2(s[2 * e + 1], v.y, a1);
                s[2 * e] = fma2(s[2 * e], ww, mul2(g.x, rr));
                s[2 * e + 1] = fma2(s[2 * e + 1], ww, mul2(g.y, rr));
            }
            const float dv = sum2(a0) + sum2(a1);
            if (live) gk_[base + (i64)t * C + i] = from_f<E>(fmaf(u * r, sm.vg[t], dv));
        }
    } else {
        const ulonglong2* wp = reinterpret_cast<const ulonglong2*>(sm.w);
        for (int t = n - 1; t >= 0; --t) {
            const float g = sm.g[t * NMAX + i];
            const f2 gg = pack2(g, g);
            const ulonglong2 *rp = reinterpret_cast<const ulonglong2*>(sm.r + t * NMAX), *kp = reinterpret_cast<const ulonglong2*>(sm.k + t * NMAX);
            f2 a0 = 0ull, a1 = 0ull;
#pragma unroll
            for (int e = 0; e < NMAX / 4; ++e) {
                const ulonglong2 r = rp[e], k = kp[e], wj = wp[e];
                a0 = fma2(s[2 * e], k.x, a0);
                a1 = fma2(s[2 * e + 1], k.y, a1);
                s[2 * e] = fma2(s[2 * e], wj.x, mul2(r.x, gg));
                s[2 * e + 1] = fma2(s[2 * e + 1], wj.y, mul2(r.y, gg));
            }
            if (live) gv_[base + (i64)t * C + i] = from_f<E>(fmaf(g, sm.ruk[t], sum2(a0) + sum2(a1)));
        }
    }
}

template <typename E, int NMAX>
int forward(int B, int T, int C, int H, const void* r, const void* k, const void* v, const void* w, const void* u, void* y, float* states,
            cudaStream_t st) {
    const int N = C / H, nseg = (T + kSeg - 1) / kSeg;
    const dim3 grid(nseg, B * H), scan((N * N + 255) / 256, B * H);
    seg_local_kernel<E, NMAX, false><<<grid, NMAX, 0, st>>>(T, C, H, N, (const E*)k, (const E*)v, (const E*)w, states);
    seg_scan_kernel<E, false><<<scan, 256, 0, st>>>(T, H, N, nseg, (const E*)w, states);
    seg_y_kernel<E, NMAX><<<grid, NMAX, 0, st>>>(T, C, H, N, (const E*)r, (const E*)k, (const E*)v, (const E*)w, (const E*)u, states, (E*)y);
    return check_launch("wkv5_train_forward(segments)");
}

template <typename E, int NMAX>
int backward(int B, int T, int C, int H, const void* r, const void* k, const void* v, const void* w, const void* u, const void* gy, void* gr,
             void* gk, void* gv, const float* S, float* D, float* partial, cudaStream_t st) {
    const int N = C / H, nseg = (T + kSeg - 1) / kSeg, smem = sizeof(BwdSmem<NMAX>);
    const dim3 grid(nseg, B * H), scan((N * N + 255) / 256, B * H);
    const cudaError_t e = cudaFuncSetAttribute(seg_backward_kernel<E, NMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    RWKV_REQUIRE(e == cudaSuccess, RWKVB200_ECUDA, "wkv5_train_backward: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    seg_local_kernel<E, NMAX, true><<<grid, NMAX, 0, st>>>(T, C, H, N, (const E*)r, (const E*)gy, (const E*)w, D);
    seg_scan_kernel<E, true><<<scan, 256, 0, st>>>(T, H, N, nseg, (const E*)w, D);
    seg_backward_kernel<E, NMAX><<<grid, 4 * NMAX, smem, st>>>(T, C, H, N, (const E*)r, (const E*)k, (const E*)v, (const E*)w, (const E*)u,
                                                              (const E*)gy, S, D, (E*)gr, (E*)gk, (E*)gv, partial);
    return check_launch("wkv5_train_backward(segments)");
}

}  // namespace

#define RWKV_BY_SHAPE(CALL)                                                                     \
    switch (head_capacity(C / H)) {                                                             \
        case 32: return dtype == RWKVB200_F32 ? CALL(float, 32) : CALL(bf16, 32);               \
        case 64: return dtype == RWKVB200_F32 ? CALL(float, 64) : CALL(bf16, 64);               \
        default: return dtype == RWKVB200_F32 ? CALL(float, 128) : CALL(bf16, 128);             \
    }
int wkv5_seg_forward(int dtype, int B, int T, int C, int H, const void* r, const void* k, const void* v, const void* w, const void* u, void* y,
                     float* states, cudaStream_t st) {
#define CALL(E, NM) forward<E, NM>(B, T, C, H, r, k, v, w, u, y, states, st)
    RWKV_BY_SHAPE(CALL)
#undef CALL
}
int wkv5_seg_backward(int dtype, int B, int T, int C, int H, const void* r, const void* k, const void* v, const void* w, const void* u,
                      const void* gy, void* gr, void* gk, void* gv, const float* S, float* D, float* partial, cudaStream_t st) {
#define CALL(E, NM) backward<E, NM>(B, T, C, H, r, k, v, w, u, gy, gr, gk, gv, S, D, partial, st)
    RWKV_BY_SHAPE(CALL)
#undef CALL
}

}  // namespace rwkvb200
