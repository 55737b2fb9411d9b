// RWKV-6 training in fp32 arithmetic, bf16 activations, head size 64, no state in or out, split over time: the lengths that
// are not whole tiles of the tensor-core kernels (wkv6_seg_applies).
//
// Per (batch, head), S indexed [key j][value i], d_t[j] = exp(-exp(w_t[j])) the decay of token t:
//   y_t[i] = sum_j r_t[j] S_{t-1}[j,i] + v_t[i] sum_j r_t u k_t      S_t[j,i] = d_t[j] S_{t-1}[j,i] + k_t[j] v_t[i]
// The steps are those of wkv5_seg.cu, with the products of the token decays in place of powers of one decay:
//   states  at the start of every segment of 32 tokens (backward: the adjoint D = dL/dS behind it; k, v -> r, gy, time reversed):
//           with many units by a walk along the segments (seg_mma_chain_kernel), with few by local end states from a zero start,
//           sum_s (prod_{tau>s} d_tau) k_s v_s^T, and a scan over them in place, S <- S diag(prod d) + local.  The products of
//           decays that are put on k are <= 1: nothing can overflow, whatever the decays are;
//   y, gradients  of every segment at the same time from its states, by the products of seg_mma.cuh.  Segments that these leave
//           (decays out of range, values that are not finite) are walked token by token by the kernels here: two warps carry S
//           forward (gr) while two carry D backward (gk, gv).  For the decay gradient they leave P_t = r_t sum_i gy_t S_{t-1} and
//           Q_t = k_t sum_i D_t v_t, and with A_t = sum_i D_{t-1}[j,i] S_{t-1}[j,i] (D_t: before token t is taken in, S_t: after it)
//   dL/dlog d_t = A_{t+1} - Q_t       A_t = A_{t+1} - Q_t + P_t       (wkv6.cu)
// walked over the segment's tokens only: A at its end is taken from the two states there.
//
// B8 T1000 H32, forward + backward on a B200: 4374 us on the general-shape kernels, which walk the tokens with one block per unit;
// 1237 us with the token-by-token kernels on all segments (multiply-adds at 46 % of the issue slots and the shared-memory reads of
// the tokens' vectors); 499 us with products, 1205 us where every segment has
// a decay too strong for them.  Errors of bf16 results against fp64 are the same to four digits (1.66e-3: one rounding; B2 T1000 H40, decay inputs
// around -5 to 1).
// The kernels for whole 32-token chunks take 258 us, but their operands are TF32: outputs are then 2 to 4 % further from fp64.
#include "wkv6_seg.cuh"
#include "seg_mma.cuh"

namespace rwkvb200 {
namespace {

constexpr float kLeast = 1.f / (1ll << (int)kRange);
__device__ __forceinline__ float log_decay(const bf16* w_raw) { return -expf(to_f(*w_raw)); }

// d of the segment's tokens as rows in the order of place(); 1 where there is no token.
template <int NTH>
__device__ __forceinline__ void stage_decay(float* dst, const bf16* __restrict__ w, int n, int C, int tid) {
    stage<NTH>(dst, w, n, C, kN, tid);
    // (each element is changed by the thread that reads it here, whichever thread has staged it)
    __syncthreads();
    for (int x = tid; x < kSeg * kN; x += NTH) dst[x] = x < n * kN ? expf(-expf(dst[x])) : 1.f;
}

// In place: local end states -> state before each segment (REV: adjoint after each segment).  One thread per state element.
template <bool REV>
__global__ void __launch_bounds__(256) seg6_scan_kernel(int nseg, const float* __restrict__ decays, float* __restrict__ states) {
    const i64 unit = blockIdx.x / (kN * kN / 256);
    const int e = blockIdx.x % (kN * kN / 256) * 256 + threadIdx.x;
    const float* d = decays + unit * nseg * kN + place(e / kN);
    float* p = states + unit * nseg * kN * kN + e;
    constexpr int AHEAD = 16;
    float cur = 0.f;
    for (int k0 = 0; k0 < nseg; k0 += AHEAD) {   // the loads of AHEAD segments are in flight together
        float x[AHEAD], f[AHEAD];
#pragma unroll
        for (int q = 0; q < AHEAD; ++q)
            if (k0 + q < nseg) {
                const i64 k = REV ? nseg - 1 - k0 - q : k0 + q;
                x[q] = p[k * kN * kN];
                f[q] = d[k * kN];
            }
#pragma unroll
        for (int q = 0; q < AHEAD; ++q)
            if (k0 + q < nseg) {
                p[(i64)(REV ? nseg - 1 - k0 - q : k0 + q) * kN * kN] = cur;
                cur = fmaf(cur, f[q], x[q]);
            }
    }
}

// One block per (unit, segment), 2 warps: a warp has the keys 32 warp .. of all values, a lane 8 keys x 8 values.
// REV = false: a = k, b = v, and the product of the segment's decays goes to `decays`; REV = true: a = r, b = gy.
template <bool REV>
__global__ void __launch_bounds__(64) seg6_local_kernel(int T, int H, int nseg, const bf16* __restrict__ a_, const bf16* __restrict__ b_,
                                                        const bf16* __restrict__ w_, float* __restrict__ states, float* __restrict__ decays,
                                                        int* __restrict__ flags) {
    __shared__ __align__(16) float as[kSeg * kN], bs[kSeg * kN], ds[kSeg * kN];
    const i64 unit = blockIdx.x / nseg;
    const int seg = blockIdx.x % nseg, h = unit % H, tid = threadIdx.x, lane = tid & 31, C = H * kN;
    const int n = min(kSeg, T - seg * kSeg);
    const i64 base = (unit / H * T + (i64)seg * kSeg) * C + h * kN;
    stage<64>(as, a_ + base, n, C, kN, tid);
    stage<64>(bs, b_ + base, n, C, kN, tid);
    stage_decay<64>(ds, w_ + base, n, C, tid);
    __syncthreads();
    {   // a, times the decay between its token and the end (REV: the start) of the segment: a thread per channel
        float f = 1.f;
        bool out = false;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            float g = 1.f;
#pragma unroll 8
            for (int q = 0; q < kSeg / 2; ++q) {
                const int t = REV ? half * (kSeg / 2) + q : kSeg - 1 - half * (kSeg / 2) - q;
                const float d = ds[t * kN + tid];
                as[t * kN + tid] *= f;
                f *= d;
                if (!REV) g *= d;
            }
            out |= !(g >= kLeast);
        }
        if (!REV) decays[(i64)blockIdx.x * kN + tid] = f;
        out = __syncthreads_or(out);
        if (!REV && flags != nullptr && tid == 0) flags[blockIdx.x] = out;   // (as the products would find it, at less cost)
    }
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
    store_tile(s, states + (i64)blockIdx.x * kN * kN, 8 * kg, 8 * vg, kN);
}

// The segments that seg_mma_y_kernel has left.  2 warps: a warp has the values 32 warp .. of all keys
__device__ __forceinline__ void seg6_y_segment(i64 block, int T, int H, int nseg, const bf16* __restrict__ r_, const bf16* __restrict__ k_,
                                                    const bf16* __restrict__ v_, const bf16* __restrict__ w_, const bf16* __restrict__ u_,
                                                    const float* __restrict__ states, bf16* __restrict__ y_) {
    __shared__ __align__(16) float rs[kSeg * kN], ks[kSeg * kN], vs[kSeg * kN], ds[kSeg * kN], us[kN], ruk[kSeg];
    const i64 unit = block / nseg;
    const int seg = block % nseg, h = unit % H, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, C = H * kN;
    const int n = min(kSeg, T - seg * kSeg);
    const i64 base = (unit / H * T + (i64)seg * kSeg) * C + h * kN;
    const int kg = lane >> 2, vg = 4 * warp + (lane & 3);
    Tile s;
    load_tile(s, states + block * kN * kN, 8 * kg, 8 * vg, kN);
    stage<64>(rs, r_ + base, n, C, kN, tid);
    stage<64>(ks, k_ + base, n, C, kN, tid);
    stage<64>(vs, v_ + base, n, C, kN, tid);
    us[place(tid)] = to_f(u_[h * kN + tid]);
    stage_decay<64>(ds, w_ + base, n, C, tid);
    __syncthreads();
    for (int t = warp; t < n; t += 2) {   // the bonus of a token: one warp each
        float x = fmaf(rs[t * kN + lane] * us[lane], ks[t * kN + lane], rs[t * kN + 32 + lane] * us[32 + lane] * ks[t * kN + 32 + lane]);
#pragma unroll
        for (int m = 16; m; m >>= 1) x += __shfl_xor_sync(0xffffffffu, x, m);
        if (lane == 0) ruk[t] = x;
    }
    __syncthreads();
    const int i_out = 8 * vg + kg;   // the value whose sum this lane ends with
    for (int t = 0; t < n; ++t) {
        f2 r[4], k[4], d[4], v[8];
        pairs(load8(rs + t * kN, kg), r);
        pairs(load8(ks + t * kN, kg), k);
        pairs(load8(ds + t * kN, kg), d);
        twice(load8(vs + t * kN, vg), v);
        float y[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            f2 acc = mul2(s[i][0], r[0]);
#pragma unroll
            for (int p = 1; p < 4; ++p) acc = fma2(s[i][p], r[p], acc);
#pragma unroll
            for (int p = 0; p < 4; ++p) s[i][p] = fma2(s[i][p], d[p], mul2(k[p], v[i]));
            y[i] = sum2(acc);
        }
        const float yo = reduce8(y, lane);
        y_[base + (i64)t * C + i_out] = from_f<bf16>(fmaf(vs[t * kN + place(i_out)], ruk[t], yo));
    }
}

template <bool ONE>
__global__ void __launch_bounds__(64, ONE ? 1 : 6) seg6_y_kernel(int T, int H, int nseg, const bf16* __restrict__ r_, const bf16* __restrict__ k_,
                                                    const bf16* __restrict__ v_, const bf16* __restrict__ w_, const bf16* __restrict__ u_,
                                                    const float* __restrict__ states, bf16* __restrict__ y_, const int* __restrict__ flags, i64 total) {
    for_flagged<ONE>(flags, total, [&](i64 block) { seg6_y_segment(block, T, H, nseg, r_, k_, v_, w_, u_, states, y_); });
}

// The segments that seg_mma_backward_kernel has left.  4 warps: warps 0, 1 carry S forward (gr, gu, P), warps 2, 3 carry D backward (gk, gv, Q); a warp
// has 32 keys of all values.  gv sums over all keys: the two halves meet in shared memory at the end.
struct Bwd6Smem {
    float r[kSeg * kN], k[kSeg * kN], v[kSeg * kN], g[kSeg * kN], d[kSeg * kN], gv[2][kSeg * kN];
    float P[kSeg * kN], Q[kSeg * kN], A[kN];   // [token][channel]
    float u[kN], vg[kSeg], ruk[kSeg];
};

__device__ __forceinline__ void seg6_backward_segment(i64 block, int T, int H, int nseg, const bf16* __restrict__ r_, const bf16* __restrict__ k_,
                                                      const bf16* __restrict__ v_, const bf16* __restrict__ w_, const bf16* __restrict__ u_,
                                                      const bf16* __restrict__ gy_, const float* __restrict__ S_, const float* __restrict__ D_,
                                                      bf16* __restrict__ gr_, bf16* __restrict__ gk_, bf16* __restrict__ gv_, bf16* __restrict__ gw_,
                                                      float* __restrict__ gu_) {
    extern __shared__ __align__(16) unsigned char smem_seg6[];
    Bwd6Smem& sm = *reinterpret_cast<Bwd6Smem*>(smem_seg6);
    const i64 unit = block / nseg;
    const int seg = block % nseg, h = unit % H, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, C = H * kN;
    const int n = min(kSeg, T - seg * kSeg);
    const i64 base = (unit / H * T + (i64)seg * kSeg) * C + h * kN;
    const float* D0 = D_ + block * kN * kN;
    const int kg = 4 * (warp & 1) + (lane & 3), vg = lane >> 2, j_out = 8 * kg + vg;   // j_out: the key whose sums this lane ends with
    Tile s;
    load_tile(s, warp < 2 ? S_ + block * kN * kN : D0, 8 * kg, 8 * vg, kN);
    stage<128>(sm.r, r_ + base, n, C, kN, tid);
    stage<128>(sm.k, k_ + base, n, C, kN, tid);
    stage<128>(sm.v, v_ + base, n, C, kN, tid);
    stage<128>(sm.g, gy_ + base, n, C, kN, tid);
    if (tid < kN) sm.u[place(tid)] = to_f(u_[h * kN + tid]);
    stage_decay<128>(sm.d, w_ + base, n, C, tid);
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
    if (warp < 2) {
        float gu = 0.f;
        for (int t = 0; t < n; ++t) {
            f2 k[4], d[4], v[8], g[8], sg[4];
            pairs(load8(sm.k + t * kN, kg), k);
            pairs(load8(sm.d + t * kN, kg), d);
            twice(load8(sm.v + t * kN, vg), v);
            twice(load8(sm.g + t * kN, vg), g);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    sg[p] = i ? fma2(s[i][p], g[i], sg[p]) : mul2(s[i][p], g[i]);
                    s[i][p] = fma2(s[i][p], d[p], mul2(k[p], v[i]));
                }
            float x[8];
#pragma unroll
            for (int p = 0; p < 4; ++p) unpack2(sg[p], x[2 * p], x[2 * p + 1]);
            const float sgj = reduce8(x, lane), rj = sm.r[t * kN + place(j_out)], kj = sm.k[t * kN + place(j_out)], vgt = sm.vg[t];
            gr_[base + (i64)t * C + j_out] = from_f<bf16>(fmaf(uj * kj, vgt, sgj));
            sm.P[t * kN + j_out] = rj * sgj;
            gu = fmaf(rj * kj, vgt, gu);
        }
        f2 a2[4] = {0ull, 0ull, 0ull, 0ull};   // A at the end: sum over values of D_end S_end
        float x[8];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            f2 e[8];
            load_pair(e, p, D0, 8 * kg, 8 * vg, kN);
#pragma unroll
            for (int i = 0; i < 8; ++i) a2[p] = fma2(e[i], s[i][p], a2[p]);
            unpack2(a2[p], x[2 * p], x[2 * p + 1]);
        }
        sm.A[j_out] = reduce8(x, lane);
        gu_[(unit / H * nseg + seg) * C + h * kN + j_out] = gu;
    } else {
        for (int t = n - 1; t >= 0; --t) {
            f2 r[4], k[4], d[4], v[8], g[8];
            pairs(load8(sm.r + t * kN, kg), r);
            pairs(load8(sm.k + t * kN, kg), k);
            pairs(load8(sm.d + t * kN, kg), d);
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
                    s[i][p] = fma2(s[i][p], d[p], mul2(r[p], g[i]));
                }
            }
#pragma unroll
            for (int p = 0; p < 4; ++p) unpack2(gk[p], x[2 * p], x[2 * p + 1]);
            const float dv = reduce8(x, lane);
            gk_[base + (i64)t * C + j_out] = from_f<bf16>(fmaf(uj * sm.r[t * kN + place(j_out)], sm.vg[t], dv));
            sm.Q[t * kN + j_out] = sm.k[t * kN + place(j_out)] * dv;
            reduce8_pairs(y, lane);
            *reinterpret_cast<float2*>(sm.gv[warp - 2] + t * kN + 8 * vg + 2 * (lane & 3)) = make_float2(y[0], y[1]);
        }
    }
    __syncthreads();
    if (warp < 2) {   // the decay gradient: a thread per channel
        float A = sm.A[tid];
        for (int t = n - 1; t >= 0; --t) {
            const i64 o = base + (i64)t * C + tid;
            A -= sm.Q[t * kN + tid];
            gw_[o] = from_f<bf16>(A * log_decay(w_ + o));   // d log d / d w_raw = log d
            A += sm.P[t * kN + tid];
        }
    } else {
        const int i = tid - 64;
        for (int t = 0; t < n; ++t)
            gv_[base + (i64)t * C + i] = from_f<bf16>(fmaf(sm.g[t * kN + place(i)], sm.ruk[t], sm.gv[0][t * kN + i] + sm.gv[1][t * kN + i]));
    }
}

template <bool ONE>
__global__ void __launch_bounds__(128, 3) seg6_backward_kernel(int T, int H, int nseg, const bf16* __restrict__ r_, const bf16* __restrict__ k_,
                                                               const bf16* __restrict__ v_, const bf16* __restrict__ w_,
                                                               const bf16* __restrict__ u_, const bf16* __restrict__ gy_,
                                                               const float* __restrict__ S_, const float* __restrict__ D_, bf16* __restrict__ gr_,
                                                               bf16* __restrict__ gk_, bf16* __restrict__ gv_, bf16* __restrict__ gw_,
                                                               float* __restrict__ gu_, const int* __restrict__ flags, i64 total) {
    for_flagged<ONE>(flags, total, [&](i64 block) { seg6_backward_segment(block, T, H, nseg, r_, k_, v_, w_, u_, gy_, S_, D_, gr_, gk_, gv_, gw_, gu_); });
}

}  // namespace

int wkv6_seg_forward(int B, int T, int H, const void* r, const void* k, const void* v, const void* w, const void* u, void* y, float* saved,
                     cudaStream_t st) {
    const int nseg = (T + kSeg - 1) / kSeg;
    const i64 units = (i64)B * H, total = units * nseg;
    RWKV_REQUIRE(total < (1ll << 31), RWKVB200_EINVAL, "wkv6_train_forward: too many segments");
    float* decays = saved + total * kN * kN;
    int* flags = seg_mma_pays(total) ? reinterpret_cast<int*>(decays + total * kN) : nullptr;
    if (seg_chain_pays(units)) {
        if (const int e = seg_chain<bf16, false, false>(units, T, H, nseg, k, v, w, saved, nullptr, st)) return e;
    } else {
        seg6_local_kernel<false><<<(unsigned)total, 64, 0, st>>>(T, H, nseg, (const bf16*)k, (const bf16*)v, (const bf16*)w, saved, decays, flags);
        seg6_scan_kernel<false><<<(unsigned)(units * (kN * kN / 256)), 256, 0, st>>>(nseg, decays, saved);
    }
    if (flags != nullptr)
        if (const int e = seg_mma_y<bf16, false>(total, T, H, nseg, r, k, v, w, u, saved, y, flags, !seg_chain_pays(units), st)) return e;
    const bool one = flags == nullptr || block_per_segment(total, 6);
    (one ? seg6_y_kernel<true> : seg6_y_kernel<false>)<<<(unsigned)(one ? total : 4 * resident_blocks(6)), 64, 0, st>>>(
        T, H, nseg, (const bf16*)r, (const bf16*)k, (const bf16*)v, (const bf16*)w, (const bf16*)u, saved, (bf16*)y, flags, total);
    return check_launch("wkv6_train_forward(segments)");
}

int wkv6_seg_backward(int B, int T, int H, const void* r, const void* k, const void* v, const void* w, const void* u, const void* gy, void* gr,
                      void* gk, void* gv, void* gw, const float* saved, float* adjoints, float* gu_partial, int* flags, cudaStream_t st) {
    const int nseg = (T + kSeg - 1) / kSeg;
    const i64 units = (i64)B * H, total = units * nseg;
    const float* decays = saved + total * kN * kN;
    const int* left = seg_chain_pays(units) ? nullptr : reinterpret_cast<const int*>(decays + total * kN);   // known from the forward
    const bool one = !seg_mma_pays(total) || block_per_segment(total, 3);
    const cudaError_t e = one ? allow_smem<seg6_backward_kernel<true>>(sizeof(Bwd6Smem)) : allow_smem<seg6_backward_kernel<false>>(sizeof(Bwd6Smem));
    RWKV_REQUIRE(e == cudaSuccess, RWKVB200_ECUDA, "wkv6_train_backward: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    if (seg_chain_pays(units)) {
        if (const int e = seg_chain<bf16, false, true>(units, T, H, nseg, r, gy, w, adjoints, nullptr, st)) return e;
    } else {
        seg6_local_kernel<true><<<(unsigned)total, 64, 0, st>>>(T, H, nseg, (const bf16*)r, (const bf16*)gy, (const bf16*)w, adjoints, nullptr, nullptr);
        seg6_scan_kernel<true><<<(unsigned)(units * (kN * kN / 256)), 256, 0, st>>>(nseg, decays, adjoints);
    }
    if (!seg_mma_pays(total)) flags = nullptr;
    else if (const int e = seg_mma_backward<bf16, false>(total, T, H, nseg, r, k, v, w, u, gy, saved, adjoints, gr, gk, gv, gw, gu_partial, left, flags, st)) return e;
    (one ? seg6_backward_kernel<true> : seg6_backward_kernel<false>)<<<(unsigned)(one ? total : 4 * resident_blocks(3)), 128, sizeof(Bwd6Smem), st>>>(
        T, H, nseg, (const bf16*)r, (const bf16*)k, (const bf16*)v, (const bf16*)w, (const bf16*)u, (const bf16*)gy, saved, adjoints, (bf16*)gr, (bf16*)gk,
        (bf16*)gv, (bf16*)gw, gu_partial, flags, total);
    return check_launch("wkv6_train_backward(segments)");
}

}  // namespace rwkvb200
