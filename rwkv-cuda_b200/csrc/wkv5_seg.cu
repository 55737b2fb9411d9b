// RWKV-5 training in fp32 arithmetic (fp32 activations; bf16 where the tensor-core kernels do not apply), head sizes
// N <= 64, split over time.
//
// Per (batch, head), S indexed [key j][value i], w the decay of a key:
//   y_t[i] = sum_j r_t[j] S_{t-1}[j,i] + v_t[i] sum_j r_t u k_t      S_t[j,i] = w[j] S_{t-1}[j,i] + k_t[j] v_t[i]
// wkv5.cu walks T tokens with one thread per state line: 0.4 to 0.9 us per token and sweep, with 8 to 128 units for 148 SMs.
// The state is linear in its start, so T is cut into segments of kSeg tokens which are all worked on at the same time:
//   local   the end state of every segment from a zero start: sum_s w^{n-1-s} k_s v_s^T, one multiply-add per state element
//           and token because the powers of w are put on k when it is staged (they are <= 1: nothing can overflow, whatever w is);
//   scan    start states of the segments, in place: S <- S diag(w^n) + local;
//   y       every segment again, token by token from its start state.
// Backward: the same two steps for the adjoint D = dL/dS (k, v -> r, gy, time reversed), then one block per segment: two warps
// carry S forward (gr) while two carry D backward (gk, gv).
// The decays of a segment act on its own outputs and on its end state: with Z = dS/dlog w counted from the segment's start
// (Z_0 = 0, Z <- w (Z + S)), the segment's part of dL/dlog w is sum_t r_t sum_i gy_t Z_t + sum_i D_end Z_end.  (The sum over
// states and gradients that needs no Z cancels for fast decays: 10 % error in gw at w = exp(-exp(3)).)
// With head size 64 the states come from one block per unit that walks its segments where there are many units, and y and the
// gradients from products of split operands (seg_mma.cuh); the kernels here then take the segments that those leave, and all of them
// for smaller heads and in small launches.
// Their inputs are staged in shared memory once per segment, so the token loops have no barrier; multiply-adds are packed in pairs.
// Shared memory delivers 4 bytes per lane and clock even when all lanes read the same word, so with one state line per thread
// the reads of the token's vectors bound everything (512 bytes per 96 packed multiply-adds); a lane therefore owns a tile of
// 8 keys x 8 values, and the sums over lanes are taken for eight elements at a time (7 shuffles).
// fp32, B8 T512 H16 N64, forward + backward on a B200: 1285 us with wkv5.cu, 309 us token by token on all segments (without register
// spills in the backward, which two blocks per SM allow and three do not: 212 -> 167 us for that kernel), 190 us by products, whose errors
// against fp64 are a third of that (T 1000, w from -6 to -1: y 5.2e-7 -> 1.8e-7 of the norm, gw 9.2e-7 -> 2.9e-7), 278 us where every head is
// left to the kernels here.
#include "wkv5_seg.cuh"
#include "seg_mma.cuh"

namespace rwkvb200 {
namespace {

static_assert(kSeg == kWkv5Seg, "tokens of a segment");

template <typename E>
__device__ __forceinline__ float log_decay(const E* w_raw) { return -expf(to_f(*w_raw)); }   // log w = -exp(w_raw)
__device__ __forceinline__ float power(float lw, int e) { return e == 0 ? 1.f : expf(lw * (float)e); }   // w^e, also for w = 0

// In place: local end states -> state before each segment (REV: adjoint after each segment).  One thread per state element.
template <typename E, bool REV>
__global__ void __launch_bounds__(256) seg_scan_kernel(int T, int H, int N, int nseg, const E* __restrict__ w_, float* __restrict__ states) {
    const int parts = (N * N + 255) / 256, unit = blockIdx.x / parts, e = blockIdx.x % parts * 256 + threadIdx.x;
    if (e >= N * N) return;
    const float lw = log_decay(w_ + (unit % H) * N + e / N);
    const float full = expf(lw * kSeg), tail = expf(lw * (float)(T - (nseg - 1) * kSeg));
    float* p = states + (i64)unit * nseg * N * N + e;
    constexpr int AHEAD = 16;
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

// One block per (unit, segment), 2 warps: a warp has the keys 32 warp .. of all values, a lane 8 keys x 8 values.
// REV = false: a = k, b = v; REV = true: a = r, b = gy.
template <typename E, bool REV>
__global__ void __launch_bounds__(64, 8) seg_local_kernel(int T, int C, int H, int N, int nseg, const E* __restrict__ a_, const E* __restrict__ b_,
                                                          const E* __restrict__ w_, float* __restrict__ states, int* __restrict__ flags) {
    __shared__ __align__(16) float as[kSeg * kN], bs[kSeg * kN], lw[kN];
    const int unit = blockIdx.x / nseg, seg = blockIdx.x % nseg, h = unit % H, tid = threadIdx.x, lane = tid & 31;
    const int n = min(kSeg, T - seg * kSeg);
    const i64 base = ((i64)(unit / H) * T + seg * kSeg) * C + h * N;
    lw[tid] = tid < N ? log_decay(w_ + h * N + tid) : 0.f;
    stage<64>(bs, b_ + base, n, C, N, tid);
    const bool out = __syncthreads_or(beyond(make_float2(kLog2e * lw[tid], 0.f), kStaticRange));
    if (!REV && flags != nullptr && tid == 0) flags[blockIdx.x] = out;
    // a, times the decay between its token and the end (REV: the start) of the segment
    stage<64>(as, a_ + base, n, C, N, tid, [&](int t, int j) { return t < n ? power(lw[j], REV ? t : n - 1 - t) : 0.f; });
    __syncthreads();
    const int kg = 4 * (tid >> 5) + (lane & 3), vg = lane >> 2;
    Tile s;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int p = 0; p < 4; ++p) s[i][p] = 0ull;
#pragma unroll 2
    for (int t = 0; t < n; ++t) {
        f2 a[4], b[8];
        pairs(load8(as + t * kN, kg), a);
        twice(load8(bs + t * kN, vg), b);
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int p = 0; p < 4; ++p) s[i][p] = fma2(a[p], b[i], s[i][p]);
    }
    store_tile(s, states + (i64)blockIdx.x * N * N, 8 * kg, 8 * vg, N);
}

// A segment token by token.  2 warps: a warp has the values 32 warp .. of all keys
template <typename E>
__device__ __forceinline__ void y_segment(i64 block, int T, int C, int H, int N, int nseg, const E* __restrict__ r_, const E* __restrict__ k_,
                                          const E* __restrict__ v_, const E* __restrict__ w_, const E* __restrict__ u_,
                                          const float* __restrict__ states, E* __restrict__ y_) {
    __shared__ __align__(16) float rs[kSeg * kN], ks[kSeg * kN], vs[kSeg * kN], ws[kN], us[kN], ruk[kSeg];
    const int unit = block / nseg, seg = block % nseg, h = unit % H, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = min(kSeg, T - seg * kSeg);
    const i64 base = ((i64)(unit / H) * T + seg * kSeg) * C + h * N;
    const int kg = lane >> 2, vg = 4 * warp + (lane & 3);
    Tile s;
    load_tile(s, states + block * N * N, 8 * kg, 8 * vg, N);
    stage<64>(rs, r_ + base, n, C, N, tid);
    stage<64>(ks, k_ + base, n, C, N, tid);
    stage<64>(vs, v_ + base, n, C, N, tid);
    ws[place(tid)] = tid < N ? expf(log_decay(w_ + h * N + tid)) : 0.f;
    us[place(tid)] = tid < N ? to_f(u_[h * N + tid]) : 0.f;
    __syncthreads();
    for (int t = warp; t < n; t += 2) {   // the bonus of a token: one warp each
        float x = fmaf(rs[t * kN + lane] * us[lane], ks[t * kN + lane], rs[t * kN + 32 + lane] * us[32 + lane] * ks[t * kN + 32 + lane]);
#pragma unroll
        for (int m = 16; m; m >>= 1) x += __shfl_xor_sync(0xffffffffu, x, m);
        if (lane == 0) ruk[t] = x;
    }
    __syncthreads();
    f2 w[4];
    pairs(load8(ws, kg), w);
    const int i_out = 8 * vg + kg;   // the value whose sum this lane ends with
    for (int t = 0; t < n; ++t) {
        f2 r[4], k[4], v[8];
        pairs(load8(rs + t * kN, kg), r);
        pairs(load8(ks + t * kN, kg), k);
        twice(load8(vs + t * kN, vg), v);
        float y[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            f2 acc = mul2(s[i][0], r[0]);
#pragma unroll
            for (int p = 1; p < 4; ++p) acc = fma2(s[i][p], r[p], acc);
#pragma unroll
            for (int p = 0; p < 4; ++p) s[i][p] = fma2(s[i][p], w[p], mul2(k[p], v[i]));
            y[i] = sum2(acc);
        }
        const float yo = reduce8(y, lane);
        if (i_out < N) y_[base + (i64)t * C + i_out] = from_f<E>(fmaf(vs[t * kN + place(i_out)], ruk[t], yo));
    }
}

// every segment, or (flags) those that the kernels by products have left
template <typename E, bool ONE>
__global__ void __launch_bounds__(64, 8) seg_y_kernel(int T, int C, int H, int N, int nseg, const E* __restrict__ r_, const E* __restrict__ k_,
                                                      const E* __restrict__ v_, const E* __restrict__ w_, const E* __restrict__ u_,
                                                      const float* __restrict__ states, E* __restrict__ y_, const int* __restrict__ flags, i64 total) {
    for_flagged<ONE>(flags, total, [&](i64 block) { y_segment(block, T, C, H, N, nseg, r_, k_, v_, w_, u_, states, y_); });
}

// A segment token by token.  4 warps: warps 0, 1 carry S and Z forward (gr, gw, gu), warps 2, 3 carry D backward (gk, gv); a warp
// has 32 keys of all values.  gv sums over all keys: the two halves meet in shared memory at the end.
struct BwdSmem {
    float r[kSeg * kN], k[kSeg * kN], v[kSeg * kN], g[kSeg * kN], gv[2][kSeg * kN];
    float w[kN], u[kN], vg[kSeg], ruk[kSeg];
};

template <typename E>
__device__ __forceinline__ void backward_segment(i64 block, int T, int C, int H, int N, int nseg, const E* __restrict__ r_, const E* __restrict__ k_,
                                                 const E* __restrict__ v_, const E* __restrict__ w_, const E* __restrict__ u_,
                                                 const E* __restrict__ gy_, const float* __restrict__ S_, const float* __restrict__ D_,
                                                 E* __restrict__ gr_, E* __restrict__ gk_, E* __restrict__ gv_, float* __restrict__ partial_) {
    extern __shared__ __align__(16) unsigned char smem_seg[];
    BwdSmem& sm = *reinterpret_cast<BwdSmem*>(smem_seg);
    const int unit = block / nseg, seg = block % nseg, h = unit % H, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = min(kSeg, T - seg * kSeg);
    const i64 base = ((i64)(unit / H) * T + seg * kSeg) * C + h * N;
    const float* D0 = D_ + block * N * N;
    const int kg = 4 * (warp & 1) + (lane & 3), vg = lane >> 2, j_out = 8 * kg + vg;   // j_out: the key whose sums this lane ends with
    Tile s;
    load_tile(s, warp < 2 ? S_ + block * N * N : D0, 8 * kg, 8 * vg, N);
    stage<128>(sm.r, r_ + base, n, C, N, tid);
    stage<128>(sm.k, k_ + base, n, C, N, tid);
    stage<128>(sm.v, v_ + base, n, C, N, tid);
    stage<128>(sm.g, gy_ + base, n, C, N, tid);
    if (tid < kN) {
        sm.w[place(tid)] = tid < N ? expf(log_decay(w_ + h * N + tid)) : 0.f;
        sm.u[place(tid)] = tid < N ? to_f(u_[h * N + tid]) : 0.f;
    }
    __syncthreads();
    for (int t = warp; t < n; t += 4) {   // sums of a token over its channels: one warp each
        const float *r = sm.r + t * kN, *k = sm.k + t * kN, *v = sm.v + t * kN, *g = sm.g + t * kN;
        float x = fmaf(r[lane] * sm.u[lane], k[lane], r[lane + 32] * sm.u[lane + 32] * k[lane + 32]);
        float z = fmaf(v[lane], g[lane], v[lane + 32] * g[lane + 32]);
#pragma unroll
        for (int m = 16; m; m >>= 1) { x += __shfl_xor_sync(0xffffffffu, x, m); z += __shfl_xor_sync(0xffffffffu, z, m); }
        if (lane == 0) { sm.ruk[t] = x; sm.vg[t] = z; }
    }
    __syncthreads();
    const float uj = sm.u[place(j_out)];
    f2 w[4];
    pairs(load8(sm.w, kg), w);
    if (warp < 2) {
        Tile z;
        f2 gw2[4] = {0ull, 0ull, 0ull, 0ull};
        float gu = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int p = 0; p < 4; ++p) z[i][p] = 0ull;
        for (int t = 0; t < n; ++t) {
            f2 r[4], k[4], v[8], g[8];
            pairs(load8(sm.r + t * kN, kg), r);
            pairs(load8(sm.k + t * kN, kg), k);
            twice(load8(sm.v + t * kN, vg), v);
            twice(load8(sm.g + t * kN, vg), g);
            f2 sg[4], zg[4];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    sg[p] = i ? fma2(s[i][p], g[i], sg[p]) : mul2(s[i][p], g[i]);
                    zg[p] = i ? fma2(z[i][p], g[i], zg[p]) : mul2(z[i][p], g[i]);
                    s[i][p] = mul2(s[i][p], w[p]);
                    z[i][p] = fma2(z[i][p], w[p], s[i][p]);
                    s[i][p] = fma2(k[p], v[i], s[i][p]);
                }
            float x[8];
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                gw2[p] = fma2(zg[p], r[p], gw2[p]);
                unpack2(sg[p], x[2 * p], x[2 * p + 1]);
            }
            const float sgj = reduce8(x, lane), rj = sm.r[t * kN + place(j_out)], kj = sm.k[t * kN + place(j_out)], vgt = sm.vg[t];
            if (j_out < N) gr_[base + (i64)t * C + j_out] = from_f<E>(fmaf(uj * kj, vgt, sgj));
            gu = fmaf(rj * kj, vgt, gu);
        }
        float x[8];   // + sum over values of D_end Z_end
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            f2 d[8];
            load_pair(d, p, D0, 8 * kg, 8 * vg, N);
#pragma unroll
            for (int i = 0; i < 8; ++i) gw2[p] = fma2(d[i], z[i][p], gw2[p]);
            unpack2(gw2[p], x[2 * p], x[2 * p + 1]);
        }
        const float gw = reduce8(x, lane);
        if (j_out < N) {
            float* p = partial_ + ((i64)(unit / H) * nseg + seg) * 2 * C + h * N + j_out;
            p[0] = log_decay(w_ + h * N + j_out) * gw;   // d log w / d w_raw = log w
            p[C] = gu;
        }
    } else {
        for (int t = n - 1; t >= 0; --t) {
            f2 r[4], k[4], v[8], g[8];
            pairs(load8(sm.r + t * kN, kg), r);
            pairs(load8(sm.k + t * kN, kg), k);
            twice(load8(sm.v + t * kN, vg), v);
            twice(load8(sm.g + t * kN, vg), g);
            f2 gk[4];
            float x[8], y[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                f2 acc = mul2(s[i][0], k[0]);
#pragma unroll
                for (int p = 1; p < 4; ++p) acc = fma2(s[i][p], k[p], acc);
                y[i] = sum2(acc);
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    gk[p] = i ? fma2(s[i][p], v[i], gk[p]) : mul2(s[i][p], v[i]);
                    s[i][p] = fma2(s[i][p], w[p], mul2(r[p], g[i]));
                }
            }
#pragma unroll
            for (int p = 0; p < 4; ++p) unpack2(gk[p], x[2 * p], x[2 * p + 1]);
            const float dv = reduce8(x, lane);
            if (j_out < N) gk_[base + (i64)t * C + j_out] = from_f<E>(fmaf(uj * sm.r[t * kN + place(j_out)], sm.vg[t], dv));
            reduce8_pairs(y, lane);
            *reinterpret_cast<float2*>(sm.gv[warp - 2] + t * kN + 8 * vg + 2 * (lane & 3)) = make_float2(y[0], y[1]);
        }
    }
    __syncthreads();
    for (int x = tid; x < n * kN; x += 128) {
        const int t = x / kN, i = x % kN;
        if (i < N) gv_[base + (i64)t * C + i] = from_f<E>(fmaf(sm.g[t * kN + place(i)], sm.ruk[t], sm.gv[0][x] + sm.gv[1][x]));
    }
}

template <typename E, bool ONE>
__global__ void __launch_bounds__(128, 2) seg_backward_kernel(int T, int C, int H, int N, int nseg, const E* __restrict__ r_, const E* __restrict__ k_,
                                                              const E* __restrict__ v_, const E* __restrict__ w_, const E* __restrict__ u_,
                                                              const E* __restrict__ gy_, const float* __restrict__ S_, const float* __restrict__ D_,
                                                              E* __restrict__ gr_, E* __restrict__ gk_, E* __restrict__ gv_,
                                                              float* __restrict__ partial_, const int* __restrict__ flags, i64 total) {
    for_flagged<ONE>(flags, total, [&](i64 block) { backward_segment(block, T, C, H, N, nseg, r_, k_, v_, w_, u_, gy_, S_, D_, gr_, gk_, gv_, partial_); });
}

// Head size 64: y and gradients by products (seg_mma.cuh), the kernels here only for the segments that those leave (flags).
template <typename E>
int forward(int B, int T, int C, int H, const void* r, const void* k, const void* v, const void* w, const void* u, void* y, float* states,
            int* flags, cudaStream_t st) {
    const int N = C / H, nseg = (T + kSeg - 1) / kSeg;
    const i64 units = B * (i64)H, total = units * nseg;
    if (N != kN || !seg_mma_pays(total)) flags = nullptr;
    if (N == kN && seg_chain_pays(units)) {
        if (const int e = seg_chain<E, true, false>(units, T, H, nseg, k, v, w, states, flags, st)) return e;
    } else {
        seg_local_kernel<E, false><<<(unsigned)total, 64, 0, st>>>(T, C, H, N, nseg, (const E*)k, (const E*)v, (const E*)w, states, flags);
        seg_scan_kernel<E, false><<<(unsigned)(units * ((N * N + 255) / 256)), 256, 0, st>>>(T, H, N, nseg, (const E*)w, states);
    }
    if (flags != nullptr)
        if (const int e = seg_mma_y<E, true>(total, T, H, nseg, r, k, v, w, u, states, y, flags, true, st)) return e;
    const bool one = flags == nullptr || block_per_segment(total, 8);
    (one ? seg_y_kernel<E, true> : seg_y_kernel<E, false>)<<<(unsigned)(one ? total : 4 * resident_blocks(8)), 64, 0, st>>>(
        T, C, H, N, nseg, (const E*)r, (const E*)k, (const E*)v, (const E*)w, (const E*)u, states, (E*)y,
                                         flags, total);
    return check_launch("wkv5_train_forward(segments)");
}

template <typename E>
int backward(int B, int T, int C, int H, const void* r, const void* k, const void* v, const void* w, const void* u, const void* gy, void* gr,
             void* gk, void* gv, const float* S, float* D, float* partial, const int* left, int* flags, cudaStream_t st) {
    const int N = C / H, nseg = (T + kSeg - 1) / kSeg, smem = sizeof(BwdSmem);
    const i64 units = B * (i64)H, total = units * nseg;
    const bool one = N != kN || !seg_mma_pays(total) || block_per_segment(total, 2);
    const cudaError_t e = one ? allow_smem<seg_backward_kernel<E, true>>(smem) : allow_smem<seg_backward_kernel<E, false>>(smem);
    RWKV_REQUIRE(e == cudaSuccess, RWKVB200_ECUDA, "wkv5_train_backward: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    if (N == kN && seg_chain_pays(units)) {
        if (const int e = seg_chain<E, true, true>(units, T, H, nseg, r, gy, w, D, nullptr, st)) return e;
    } else {
        seg_local_kernel<E, true><<<(unsigned)total, 64, 0, st>>>(T, C, H, N, nseg, (const E*)r, (const E*)gy, (const E*)w, D, nullptr);
        seg_scan_kernel<E, true><<<(unsigned)(units * ((N * N + 255) / 256)), 256, 0, st>>>(T, H, N, nseg, (const E*)w, D);
    }
    if (N != kN || !seg_mma_pays(total)) flags = nullptr;
    else if (const int e = seg_mma_backward<E, true>(total, T, H, nseg, r, k, v, w, u, gy, S, D, gr, gk, gv, nullptr, partial, left, flags, st)) return e;
    (one ? seg_backward_kernel<E, true> : seg_backward_kernel<E, false>)<<<(unsigned)(one ? total : 4 * resident_blocks(2)), 128, smem, st>>>(
        T, C, H, N, nseg, (const E*)r, (const E*)k, (const E*)v, (const E*)w, (const E*)u, (const E*)gy, S,
                                                    D, (E*)gr, (E*)gk, (E*)gv, partial, flags, total);
    return check_launch("wkv5_train_backward(segments)");
}

}  // namespace

int wkv5_seg_forward(int dtype, int B, int T, int C, int H, const void* r, const void* k, const void* v, const void* w, const void* u, void* y,
                     float* states, int* flags, cudaStream_t st) {
    return dtype == RWKVB200_F32 ? forward<float>(B, T, C, H, r, k, v, w, u, y, states, flags, st)
                                 : forward<bf16>(B, T, C, H, r, k, v, w, u, y, states, flags, st);
}
int wkv5_seg_backward(int dtype, int B, int T, int C, int H, const void* r, const void* k, const void* v, const void* w, const void* u,
                      const void* gy, void* gr, void* gk, void* gv, const float* S, float* D, float* partial, const int* left, int* flags, cudaStream_t st) {
    return dtype == RWKVB200_F32 ? backward<float>(B, T, C, H, r, k, v, w, u, gy, gr, gk, gv, S, D, partial, left, flags, st)
                                 : backward<bf16>(B, T, C, H, r, k, v, w, u, gy, gr, gk, gv, S, D, partial, left, flags, st);
}

}  // namespace rwkvb200
