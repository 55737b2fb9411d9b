// RWKV-6 / RWKV-5 forward, head size 64, bf16 activations, 32-token chunks on tcgen05: three warp groups on
// consecutive chunks, inputs by TMA (the structure of wkv7_l32_fwd_pipe.cu without the delta-rule terms).
//
// Per (batch, head), S indexed [value i][key j], d_t the decay of token t (per key channel):
//   y_t = S_{t-1} r_t + (sum_j r_t u k_t) v_t ;   S_t = S_{t-1} diag(d_t) + v_t k_t^T
// (wkv6/cuda/wkv6_cuda_v1.cu:15-66, wkv6_state/cuda/wkv6state_cuda_v1a.cu, wkv5_bf16/cuda/wkv5_cuda_v1b.cu:12-60
// of the reference project).  Within a chunk of L = 32 tokens let P_t = prod_{tau<=t} d_tau, P_{-1} = 1,
// We = P_31, and
//   r~_t = r_t P_{t-1}     k~_s = k_s / P_s     k^_s = u k_s / P_{s-1}
//   A[s,t] = k~_s . r~_t (s < t),   A[t,t] = k^_t . r~_t = sum_j r_t u k_t,   0 otherwise
// then with S0 the state at the start of the chunk and V = [v_t]:
//   Y = S0 R~^T + V A            S_end = (S0 + V K~) diag(We)
// All products are tcgen05.mma kind::tf32 (M = 64): the 64 x 32 product [K~;K^] R~^T gives the strict part
// of A in its rows 0-31 and the diagonal in the diagonal of its rows 32-63.  The divisions by P are safe while
// the summed |log d| of a chunk stays below 80; beyond that the kernel raises the flag of its (batch, head)
// unit and the general-shape kernel redoes that unit.
//
// The state in tensor memory is not scaled by We at the end of every chunk.  It is kept divided by D = the decay since
// it was last scaled, and the chunk's vectors carry D instead: r~_t = r_t D P_{t-1}, k~_s = k_s / (D P_s), so that
//   X = S^ R~^T   and   S^ += V K~
// need no pass over the state in between; A is the same.  Only when D would fall below 2^-60 (kRenormLog2: the
// exponents then keep 18 bits after the point) is S^ multiplied by D before the chunk and D set to 1.
//
//   loader warps, chunk c+2:  raw rows by TMA (r, k, v and a per-token decay input), operand preparation;
//   matrix warps, chunk c+1:  [K~;K^] R~^T on the tensor core, A masked into shared memory;
//   chain warp, chunk c:      X = S^ R~^T, Y = X + V A, S^ += V K~, nothing but products;
//   output warps, chunk c:    y out;
//   state warps, chunk c+1:   the state at its start out (for a backward pass), S^ scaled where it has to be.
// B16 T4096 H64, states saved: one chain group that also wrote y and scaled the state 1248 us (2700 cycles a chunk, whatever
// the stores and loaders did); these roles with one loader group 1330, two loader groups 1140; the states through shared
// memory and bulk copies 988 (16 stores of 8 bytes per thread were a third of the shared-memory pipe, which was 75 % busy).
#include <cuda.h>

#include "wkv7_l32.cuh"
#include "wkv6_chunked.cuh"

namespace rwkvb200 {
namespace v6q {

using namespace v7x;

constexpr int GNT = 128;          // threads of a loader group, the matrix, the output and the state warps
constexpr int LTPW = 8;           // tokens of a loader warp
constexpr int PNT = 5 * GNT + 32;
constexpr int NA = 3;             // operand sets in flight
constexpr int NU = 2;             // A matrices in flight
constexpr float kMaxChunkLog2Decay = 80.f * 1.4426950408889634f;
constexpr float kRenormLog2 = -60.f;

template <int WMODE>
struct Smem {
    static constexpr int NS = WMODE == 0 ? 2 : 4;          // chunks of raw input rows in flight, half of them per loader group
    static constexpr int kRawStage = 3 * 4096 + (WMODE == 0 ? 8192 : WMODE == 1 ? 4096 : 0);   // r, k, v tiles (bf16), the decay tile (bf16 or fp32)
    static constexpr int kASet = ARR32 + ARR64 + ARR32;   // R~ [32][64], K~ and K^ [64][64] in turns of 8 rows, V [32][64]
    static constexpr int kU = NA * kASet;                 // A matrices, swizzled [32][32]
    static constexpr int kWe = kU + NU * HALF32;          // per set: [64] S^ -> state, [64] what scales S^; then [64] of the end
    static constexpr int kHs = kWe + NA * 512 + 256;      // per group 2 x [4][64]: sums of a loader warp's decays
    static constexpr int kB = kHs + 4 * 1024;             // per group [64]: log2 D at the end of its chunk
    static constexpr int kY = kB + 512;                   // two staging tiles of y
    static constexpr int kRaw = (kY + 2 * 4096 + 127) / 128 * 128;
    static constexpr int kOut = (kRaw + NS * kRawStage + 1023) / 1024 * 1024;   // two images of the state on their way out
    static constexpr int kBar = kOut + 2 * ARR64;
    static constexpr int kBytes = kBar + 512 + 1024;
};
static_assert(Smem<0>::kASet % 1024 == 0 && Smem<0>::kU % 1024 == 0 && Smem<0>::kRaw % 128 == 0, "layout");
static_assert(Smem<0>::kBytes <= 232448 && Smem<1>::kBytes <= 232448, "one block per SM");

__device__ int g_v6q_error = 0;

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, int bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_tile(void* dst_smem, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                     smem_u32(dst_smem)),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void mbar_init_count(uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

struct Maps {
    CUtensorMap m[4];   // r, k, v (B*T, C) bf16; the decay input (B*T, C) bf16 or fp32 (unused for a static decay)
};

// arrivals: kFullA one per loader warp; kEmptyA the matrix group, the state warps and the product S^ += V K~
enum { kFullA = 0, kEmptyA = kFullA + NA, kFullU = kEmptyA + NA, kEmptyU = kFullU + NU, kFU = kEmptyU + NU, kBX, kBS, kState,
       kD, kBY = kD + 2, kYTaken = kBY + 2, kRawFull = kYTaken + 2, kNBar = kRawFull + 4 };
static_assert(8 * kNBar + 4 + 4 * (9 + NA) <= 512, "barrier space");

// WMODE: 0 = fp32 log-decay (B,T,C), 1 = bf16 raw input (B,T,C) with log-decay = -exp(w), 2 = fp32 decay value (C),
// 3 = fp32 log-decay (C)   (the forms of wkv6_chunked.cu), 4 = bf16 raw input (C) with log-decay = -exp(w)
template <int WMODE>
__global__ void __launch_bounds__(PNT, 1)
wkv6q_forward_kernel(int T, int H, const __grid_constant__ Maps maps, const void* __restrict__ wstat_, const bf16* __restrict__ u_,
                     const void* __restrict__ s0_, int s0_kind, bf16* __restrict__ y_, float* __restrict__ sT_,
                     float* __restrict__ ck_, int* __restrict__ unsafe_, int flag_div) {
    using Smem = v6q::Smem<WMODE>;
    constexpr int NS = Smem::NS, kRawStage = Smem::kRawStage;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + Smem::kBar);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + kNBar);
    volatile int* abort_word = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* gabort = abort_word + 1;                // one copy per group that decides together
    int* strong = const_cast<int*>(abort_word) + 5;       // a chunk's decay was too strong
    volatile int* renorm = reinterpret_cast<volatile int*>(strong + 1);   // per operand set: S^ is scaled before this chunk

    const int hh = blockIdx.x, bb = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int C = H * 64;
    const i64 tok0 = (i64)bb * T * C + hh * 64;
    const i64 sbase = (i64)(bb * H + hh) * 64 * 64;
    const int nchunks = (T + LC - 1) / LC;
    constexpr bool kPerToken = WMODE < 2;
    float* ck = ck_ ? ck_ + (i64)(bb * H + hh) * nchunks * 64 * 64 : nullptr;   // chunk-start states for a backward pass, as images of its operand array
    const bool states_only = y_ == nullptr;                                  // no y: the pass that only saves the states
    constexpr int kWTile = WMODE == 0 ? 8192 : 4096;

    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < kNBar; ++i)
            mbar_init_count(bar + i, i < kFullA + NA ? 4 : i < kEmptyA + NA ? 6
                                   : (i >= kFullU && i < kFullU + NU) || (i >= kD && i < kD + 2) || (i >= kYTaken && i < kYTaken + 2) || i == kState ? 4 : 1);
        *abort_word = 0; gabort[0] = 0; gabort[1] = 0; gabort[2] = 0; gabort[3] = 0; *strong = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(smem_u32(tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm0 = __shfl_sync(0xffffffffu, tmem_slot[0], 0);
    const uint32_t tmS = tm0, tmX = tm0 + 64, tmU = tm0 + 128;   // X: even and odd chunks
    const uint32_t lead = elect_one();
    const int wg = warp & 3, row0 = wg * 16;                     // the quarter of tensor memory this warp may touch
    const uint32_t lane_off = (uint32_t)(wg * 32) << 16;
    int fail = 0;

    if (warp < 8) {
        // ================================ loader warps =====================================================
        // two groups, for even and odd chunks: a chunk is one long chain of latencies for the warps that prepare it
        const int lg = warp >> 2;
        float* Hs = reinterpret_cast<float*>(smem + Smem::kHs) + lg * 512;
        float* Ds = reinterpret_cast<float*>(smem + Smem::kB);
        unsigned char* stg = smem + Smem::kRaw;
        const int j0 = 2 * lane;
        const float u0 = __bfloat162float(u_[hh * 64 + j0]), u1 = __bfloat162float(u_[hh * 64 + j0 + 1]);
        float ls0 = 0.f, ls1 = 0.f;   // log2 of a static decay
        if (WMODE == 2) {
            ls0 = __log2f(reinterpret_cast<const float*>(wstat_)[hh * 64 + j0]);
            ls1 = __log2f(reinterpret_cast<const float*>(wstat_)[hh * 64 + j0 + 1]);
        } else if (WMODE == 3) {
            ls0 = reinterpret_cast<const float*>(wstat_)[hh * 64 + j0] * 1.4426950408889634f;
            ls1 = reinterpret_cast<const float*>(wstat_)[hh * 64 + j0 + 1] * 1.4426950408889634f;
        } else if (WMODE == 4) {
            ls0 = -expf(__bfloat162float(reinterpret_cast<const bf16*>(wstat_)[hh * 64 + j0])) * 1.4426950408889634f;
            ls1 = -expf(__bfloat162float(reinterpret_cast<const bf16*>(wstat_)[hh * 64 + j0 + 1])) * 1.4426950408889634f;
        }
        int issued = 0;
        bool too_strong = false;
        auto issue_raw = [&](int c) {   // lane 0 of the group's warps issues a tile each
            const int st = c % NS;
            uint64_t* fb = bar + kRawFull + st;
            if (lane == 0) {
                if (wg == 0) mbar_expect_tx(fb, 3 * 4096 + (kPerToken ? kWTile : 0));
                if (wg < 3 || kPerToken) tma_tile(stg + st * kRawStage + wg * 4096, &maps.m[wg], hh * 64, bb * T + c * LC, fb);
            }
            issued = c + 2;
        };
        for (int cc = lg; cc < min(NS, nchunks); cc += 2) issue_raw(cc);
        int c = lg;
        for (; c < nchunks; c += 2) {
            const int valid = min(LC, T - c * LC), st = c % NS, sa = c % NA, ua = c / NA;
            unsigned char* A = smem + sa * Smem::kASet;
            unsigned char *RT = A, *KK = A + ARR32, *Vs = A + ARR32 + ARR64;
            if (!mbar_wait(bar + kRawFull + st, (c / NS) & 1)) fail = 31;
            // this thread: channels j0, j0+1 of tokens 8*wg .. 8*wg+7
            uint32_t xr[LTPW], xk[LTPW], xv[LTPW];
            float ld0[LTPW], ld1[LTPW];   // log2 decay of the token
            unsigned char* rs = stg + st * kRawStage;
            if (valid < LC) {   // the last chunk of a ragged T: neutral words in place of the rows beyond it (this thread's own)
                for (int tt = LTPW * wg; tt < LTPW * wg + LTPW; ++tt) {
                    if (tt < valid) continue;
#pragma unroll
                    for (int x = 0; x < 3; ++x) *reinterpret_cast<uint32_t*>(rs + x * 4096 + tt * 128 + 4 * lane) = 0u;
                    if (WMODE == 1) *reinterpret_cast<uint32_t*>(rs + 12288 + tt * 128 + 4 * lane) = 0xff80ff80u;   // -inf: no decay
                    if (WMODE == 0) *reinterpret_cast<float2*>(rs + 12288 + tt * 256 + 8 * lane) = make_float2(0.f, 0.f);
                }
            }
#pragma unroll
            for (int q = 0; q < LTPW; ++q) {
                const int tt = LTPW * wg + q;
                xr[q] = *reinterpret_cast<const uint32_t*>(rs + tt * 128 + 4 * lane);
                xk[q] = *reinterpret_cast<const uint32_t*>(rs + 4096 + tt * 128 + 4 * lane);
                xv[q] = *reinterpret_cast<const uint32_t*>(rs + 8192 + tt * 128 + 4 * lane);
                if (WMODE == 1) {
                    const float2 w2 = bf16x2_to_f2(*reinterpret_cast<const uint32_t*>(rs + 12288 + tt * 128 + 4 * lane));
                    ld0[q] = -fexp(w2.x) * 1.4426950408889634f;
                    ld1[q] = -fexp(w2.y) * 1.4426950408889634f;
                } else if (WMODE == 0) {
                    const float2 w2 = *reinterpret_cast<const float2*>(rs + 12288 + tt * 256 + 8 * lane);
                    ld0[q] = w2.x * 1.4426950408889634f;
                    ld1[q] = w2.y * 1.4426950408889634f;
                } else {
                    ld0[q] = tt < valid ? ls0 : 0.f;
                    ld1[q] = tt < valid ? ls1 : 0.f;
                }
            }
            // cumulative log2 decays: within the warp's tokens, then across the warps
            float cs0[LTPW], cs1[LTPW], run0 = 0.f, run1 = 0.f;
#pragma unroll
            for (int q = 0; q < LTPW; ++q) { run0 += ld0[q]; run1 += ld1[q]; cs0[q] = run0; cs1[q] = run1; }
            float* hs = Hs + ((c >> 1) & 1) * 256;
            *reinterpret_cast<float2*>(hs + wg * 64 + j0) = make_float2(run0, run1);
            if (ua >= 1 && !mbar_wait(bar + kEmptyA + sa, (ua - 1) & 1)) fail = 30;
            if (fail) atomicMax(const_cast<int*>(abort_word), fail);
            if (wg == 0 && lane == 0) gabort[lg] = *abort_word;
            proxy_fence();   // (the words are still on their way to the registers: the copy engine must not be quicker)
            group_sync(1 + lg, GNT);   // the warps' sums; every thread has taken its part of the rows, the stage may be refilled
            if (gabort[lg]) break;
            if (c + NS < nchunks) issue_raw(c + NS);
            float base0 = 0.f, base1 = 0.f, tot0 = 0.f, tot1 = 0.f;
#pragma unroll
            for (int gq = 0; gq < 4; ++gq) {
                const float2 h = *reinterpret_cast<const float2*>(hs + gq * 64 + j0);
                if (gq < wg) { base0 += h.x; base1 += h.y; }
                tot0 += h.x; tot1 += h.y;
            }
            too_strong |= -tot0 > kMaxChunkLog2Decay || -tot1 > kMaxChunkLog2Decay;
            // D at the end of the chunk before, from the other group; every warp has all channels and decides alike
            float b0 = 0.f, b1 = 0.f;
            if (c > 0) {
                if (!mbar_wait(bar + kD + (lg ^ 1), ((c - 1) >> 1) & 1)) fail = 32;
                const float2 d = *reinterpret_cast<const float2*>(Ds + (lg ^ 1) * 64 + j0);
                b0 = d.x; b1 = d.y;
            }
            const bool again = __any_sync(0xffffffffu, fminf(b0 + tot0, b1 + tot1) < kRenormLog2 && fminf(b0, b1) < 0.f);
            const float e0 = (again ? 0.f : b0) + tot0, e1 = (again ? 0.f : b1) + tot1;
            if (wg == 0) {
                *reinterpret_cast<float2*>(Ds + lg * 64 + j0) = make_float2(e0, e1);
                float* Wc = reinterpret_cast<float*>(smem + Smem::kWe + sa * 512);
                if (again) *reinterpret_cast<float2*>(Wc + 64 + j0) = make_float2(fex2(fmaxf(b0, -120.f)), fex2(fmaxf(b1, -120.f)));
                *reinterpret_cast<float2*>(Wc + j0) = again ? make_float2(1.f, 1.f) : make_float2(fex2(b0), fex2(b1));
                if (lane == 0) renorm[sa] = again;
                if (c + 1 == nchunks)   // what turns S^ into the final state
                    *reinterpret_cast<float2*>(reinterpret_cast<float*>(smem + Smem::kWe + NA * 512) + j0) =
                        make_float2(fex2(fmaxf(e0, -120.f)), fex2(fmaxf(e1, -120.f)));
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar + kD + lg);   // (all four warps: each has read what the other group will write next)
            if (again) b0 = b1 = 0.f;
            float lp0 = b0 + base0, lp1 = b1 + base1;   // log2 of the decay up to the token before
#pragma unroll
            for (int q = 0; q < LTPW; ++q) {
                const int tt = LTPW * wg + q;
                const int kr = 2 * LTPW * wg + q;   // row of k~ of this token
                // a chunk whose decay is beyond the bound is recomputed elsewhere: keep the values finite here
                const float l0 = fmaxf(b0 + base0 + cs0[q], -120.f), l1 = fmaxf(b1 + base1 + cs1[q], -120.f);
                const float p0 = fmaxf(lp0, -120.f), p1 = fmaxf(lp1, -120.f);
                const float wp0 = fex2(p0), wp1 = fex2(p1), iw0 = fex2(-l0), iw1 = fex2(-l1), ip0 = fex2(-p0), ip1 = fex2(-p1);
                const float2 r2 = bf16x2_to_f2(xr[q]), k2 = bf16x2_to_f2(xk[q]), v2 = bf16x2_to_f2(xv[q]);
                *reinterpret_cast<float2*>(RT + sw(tt, j0, HALF32)) = make_float2(tf32rf(r2.x * wp0), tf32rf(r2.y * wp1));
                *reinterpret_cast<float2*>(KK + sw(kr, j0, HALF64)) = make_float2(tf32rf(k2.x * iw0), tf32rf(k2.y * iw1));
                *reinterpret_cast<float2*>(KK + sw(kr + 8, j0, HALF64)) = make_float2(tf32rf(u0 * k2.x * ip0), tf32rf(u1 * k2.y * ip1));
                *reinterpret_cast<float2*>(Vs + sw(tt, j0, HALF32)) = v2;
                lp0 = b0 + base0 + cs0[q]; lp1 = b1 + base1 + cs1[q];
            }
            proxy_fence();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar + kFullA + sa);
        }
        if (too_strong) atomicOr(strong, 1);
        if (fail) atomicMax(const_cast<int*>(abort_word), fail);
        for (int cc = c; cc < issued; cc += 2) mbar_wait(bar + kRawFull + cc % NS, (cc / NS) & 1);   // left early: the rows asked for must have landed
    } else if (warp < 12) {
        // ================================ matrix warps =====================================================
        const int gtid = tid - 2 * GNT;
        int sa = 0, ua = 0;
        uint32_t par = 0;
        for (int c = 0; c < nchunks; ++c, par ^= 1) {
            const int su = c & 1;
            unsigned char* A = smem + sa * Smem::kASet;
            unsigned char* Am = smem + Smem::kU + su * HALF32;
            if (!mbar_wait(bar + kFullA + sa, ua & 1)) fail = 35;
            if (c >= NU && !mbar_wait(bar + kEmptyU + su, ((c >> 1) - 1) & 1)) fail = 36;
            if (fail) atomicMax(const_cast<int*>(abort_word), fail);
            if (gtid == 0) gabort[2] = *abort_word;
            tc_fence_before();
            group_sync(3, GNT);   // (and: every warp has taken the previous product out of tensor memory)
            tc_fence_after();
            if (gabort[2]) break;
            if (!states_only) {
                if (wg == 0) {   // [K~;K^] R~^T; columns = tokens t
                    const uint32_t kkA = smem_u32(A + ARR32), rtA = smem_u32(A);
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks)
                        mma_ss(tmU, desc_k(kkA, 0, ks * 8, HALF64), desc_k(rtA, 0, ks * 8, HALF32), idesc64(32, 0, 0), ks > 0, lead);
                    mma_commit(bar + kFU, lead);
                }
                if (!mbar_wait(bar + kFU, par)) fail = 37;
                tc_fence_after();
                float u[4][4];
                tmem_ld_tiles<4>(u, tmU + lane_off);
                tmem_wait_ld();
                // this warp's rows: k~_s and, 8 further down, k^_s of s = 8*wg + g; tile nt is columns 8*nt ..
                const int s = 8 * wg + g;
#pragma unroll
                for (int nt = 0; nt < 4; ++nt) {
                    const int c0 = nt * 8 + 2 * t;
                    float2 x = make_float2(tf32rf(u[nt][0]), tf32rf(u[nt][1]));
                    if (nt < wg) x = make_float2(0.f, 0.f);
                    if (nt == wg)
                        x = make_float2(s < c0 ? x.x : s == c0 ? tf32rf(u[nt][2]) : 0.f, s < c0 + 1 ? x.y : s == c0 + 1 ? tf32rf(u[nt][3]) : 0.f);
                    *reinterpret_cast<float2*>(Am + sw32(s, c0)) = x;
                }
                proxy_fence();
            }
            if (gtid == 0) mbar_arrive(bar + kEmptyA + sa);   // this group is done with the operand set
            __syncwarp();
            if (lane == 0) mbar_arrive(bar + kFullU + su);
            if (++sa == NA) { sa = 0; ++ua; }
        }
        if (fail) atomicMax(const_cast<int*>(abort_word), fail);
    } else if (warp < 16) {
        // ================================ output warps =====================================================
        const int gtid = tid - 3 * GNT;
        for (int c = 0; c < nchunks && !states_only; ++c) {
            unsigned char* stage = smem + Smem::kY + (c & 1) * 4096;
            if (!mbar_wait(bar + kBY + (c & 1), (c >> 1) & 1)) fail = 42;
            tc_fence_after();
            float Y[4][4];
            tmem_ld_tiles<4>(Y, tmX + 32 * (c & 1) + lane_off);
            tmem_wait_ld();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar + kYTaken + (c & 1));
#pragma unroll
            for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    *reinterpret_cast<bf16*>(stage + stage_off(nt * 8 + 2 * t + (e & 1), row0 + g + ((e & 2) ? 8 : 0))) = __float2bfloat16_rn(Y[nt][e]);
            if (fail) atomicMax(const_cast<int*>(abort_word), fail);
            if (gtid == 0) gabort[3] = *abort_word;
            group_sync(4, GNT);   // (and: every thread has sent its part of the chunk before, which used the other tile)
            if (gabort[3]) break;
            const int valid = min(LC, T - c * LC);
            stage_flush(stage, y_, tok0 + (i64)c * LC * C, C, gtid, valid);
            stage_flush(stage, y_, tok0 + (i64)c * LC * C, C, gtid + GNT, valid);
        }
    } else if (warp < 20) {
        // ================================ state warps ======================================================
        float Sd[8][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const i64 idx = sbase + (row0 + g + ((e & 2) ? 8 : 0)) * 64 + nt * 8 + 2 * t + (e & 1);
                Sd[nt][e] = s0_kind == 2 ? reinterpret_cast<const float*>(s0_)[idx]
                          : s0_kind == 1 ? __bfloat162float(reinterpret_cast<const bf16*>(s0_)[idx]) : 0.f;
            }
        auto scale = [&](const float* f) {   // columns of S^ times f
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                const float2 x = *reinterpret_cast<const float2*>(f + nt * 8 + 2 * t);
                Sd[nt][0] *= x.x; Sd[nt][1] *= x.y; Sd[nt][2] *= x.x; Sd[nt][3] *= x.y;
            }
        };
        int sa = 0, ua = 0, c = 0;
        for (; c < nchunks; ++c) {   // the state at the start of chunk c
            if (c > 0 && !mbar_wait(bar + kBS, (c - 1) & 1)) fail = 43;
            if (!mbar_wait(bar + kFullA + sa, ua & 1)) fail = 44;
            tc_fence_after();
            if (__any_sync(0xffffffffu, fail | *abort_word)) break;
            const float* Wc = reinterpret_cast<const float*>(smem + Smem::kWe + sa * 512);
            const bool again = __any_sync(0xffffffffu, renorm[sa]);
            if (c > 0 && (again || ck != nullptr)) {
                tmem_ld_tiles<8>(Sd, tmS + lane_off);
                tmem_wait_ld();
            }
            if (again) scale(Wc + 64);
            if (again || c == 0) {
                tmem_st_tiles<8>(tmS + lane_off, Sd);
                tmem_wait_st();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar + kState);   // the state may be read (scaled) and written (taken)
            if (ck != nullptr) {
                if (!again) scale(Wc);
                send_rows(smem + Smem::kOut, c, reinterpret_cast<unsigned char*>(ck) + (i64)c * ARR64, Sd, row0, lane);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar + kEmptyA + sa);
            if (++sa == NA) { sa = 0; ++ua; }
        }
        if (c == nchunks) {   // the final state; the last product of this block has then completed
            if (!mbar_wait(bar + kBS, (nchunks - 1) & 1)) fail = 45;
            tc_fence_after();
            if (sT_ != nullptr && !__any_sync(0xffffffffu, fail)) {
                tmem_ld_tiles<8>(Sd, tmS + lane_off);
                tmem_wait_ld();
                scale(reinterpret_cast<const float*>(smem + Smem::kWe + NA * 512));
                float* dst = sT_ + sbase;
#pragma unroll
                for (int nt = 0; nt < 8; ++nt) {
                    *reinterpret_cast<float2*>(dst + (row0 + g) * 64 + nt * 8 + 2 * t) = make_float2(Sd[nt][0], Sd[nt][1]);
                    *reinterpret_cast<float2*>(dst + (row0 + g + 8) * 64 + nt * 8 + 2 * t) = make_float2(Sd[nt][2], Sd[nt][3]);
                }
            }
        }
        sent_all(lane);
        if (fail) atomicMax(const_cast<int*>(abort_word), fail);
    } else {
        // ================================ chain warp =======================================================
        int sa = 0;
        uint32_t par = 0;
        for (int c = 0; c < nchunks; ++c, par ^= 1) {
            const int su = c & 1;
            const unsigned char* A = smem + sa * Smem::kASet;
            const uint32_t rtA = smem_u32(A), kkA = smem_u32(A + ARR32), vA = smem_u32(A + ARR32 + ARR64);
            const uint32_t amA = smem_u32(smem + Smem::kU + su * HALF32), x = tmX + 32 * su;
            if (!mbar_wait(bar + kFullU + su, (c >> 1) & 1)) fail = 40;
            const bool first = c == 0 || __any_sync(0xffffffffu, renorm[sa]);   // S^ is written before this chunk reads it
            if (first && !mbar_wait(bar + kState, par)) fail = 46;
            if (!states_only && c >= 2 && !mbar_wait(bar + kYTaken + su, ((c >> 1) - 1) & 1)) fail = 47;
            if (__any_sync(0xffffffffu, fail | *abort_word)) break;
            tc_fence_after();
            if (!states_only) {
#pragma unroll
                for (int ks = 0; ks < 8; ++ks)   // X = S^ R~^T
                    mma_ts(x, tmS + ks * 8, desc_k(rtA, 0, ks * 8, HALF32), idesc64(32, 0, 0), ks > 0, lead);
                mma_commit(bar + kBX, lead);
#pragma unroll
                for (int ks = 0; ks < 4; ++ks)   // Y = X + V A
                    mma_ss(x, desc_mn(vA, ks * 8, HALF32), desc_mn(amA, ks * 8, HALF32), idesc64(32, 1, 1), 1, lead);
                mma_commit(bar + kBY + su, lead);
                mma_commit(bar + kEmptyU + su, lead);
                if (!mbar_wait(bar + kBX, par)) fail = 41;   // X has read S^: it may be updated
            }
            if (!first && !mbar_wait(bar + kState, par)) fail = 48;
            tc_fence_after();
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)   // S^ += V K~
                mma_ss(tmS, desc_mn(vA, ks * 8, HALF32), desc_mn(kkA, ks * 16, HALF64), idesc64(64, 1, 1), 1, lead);
            mma_commit(bar + kEmptyA + sa, lead);
            if (states_only) mma_commit(bar + kEmptyU + su, lead);
            mma_commit(bar + kBS, lead);
            if (!mbar_wait(bar + kBS, par)) fail = 49;
            if (++sa == NA) sa = 0;
        }
        if (fail) atomicMax(const_cast<int*>(abort_word), fail);
    }

    tc_fence_before();
    __syncthreads();
    if (tid == 0) {   // a unit with a decay too strong for the chunked form is redone by the general-shape kernel
        if (flag_div == 0) unsafe_[bb * H + hh] = *strong;
        else if (*strong) atomicOr(unsafe_ + (((bb / flag_div) * H + hh) & (kChunkedFlagUnits - 1)), 1);
    }
    const int ab = *abort_word;
    if (ab && tid == 0) {   // a wait ran out: record it and poison this unit's outputs
        atomicMax(&g_v6q_error, ab);
        if (y_ != nullptr) y_[tok0] = __ushort_as_bfloat16((unsigned short)0x7fc0);
    }
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tm0) : "memory");
}

}  // namespace v6q

namespace {
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled6() {
    if (tensor_maps_disabled()) return nullptr;
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}
bool make_map6(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, bool fp32) {
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols * (fp32 ? 4 : 2)};
    const cuuint32_t box[2] = {64, 32};
    const cuuint32_t elem[2] = {1, 1};
    auto encode = [&] {
        return encode_tiled6()(m, fp32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims,
                               strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    // (a thread that has made no runtime call yet has no context, which this driver call wants)
    return encode() || (cudaFree(nullptr) == cudaSuccess && encode());
}
}  // namespace

bool wkv6_make_tile_map(void* map, const void* base, unsigned long long rows, unsigned long long cols, bool fp32) {
    return encode_tiled6() != nullptr && make_map6(reinterpret_cast<CUtensorMap*>(map), base, rows, cols, fp32);
}

// Returns RWKVB200_OK, an error code, or 1 when tensor maps cannot be made here (the caller then uses the
// mma.sync kernel of wkv6_chunked.cu).  Arguments as wkv6_chunked_forward; ck (optional): the states at the start of
// every 32-token chunk, (B,H,ceil(T/32),N,N) fp32, for wkv6_l32_backward; y may then be NULL (states only).
int wkv6_l32_forward(int B, int T, int H, const void* r, const void* k, const void* v, const void* w, int w_mode, const void* u,
                     const void* s0, int s0_kind, void* y, float* sT, float* ck, int* unsafe, cudaStream_t st, int flag_div) {
    using namespace v6q;
    if (encode_tiled6() == nullptr) return 1;
    Maps maps;
    const void* in[3] = {r, k, v};
    for (int x = 0; x < 3; ++x)
        if (!make_map6(&maps.m[x], in[x], (uint64_t)B * T, (uint64_t)H * 64, false)) return 1;
    if (w_mode < 2) {
        if (!make_map6(&maps.m[3], w, (uint64_t)B * T, (uint64_t)H * 64, w_mode == 0)) return 1;
    } else {
        maps.m[3] = maps.m[0];
    }
    dim3 grid(H, B);
#define RWKV_GO(M)                                                                                                       \
    do {                                                                                                                 \
        cudaError_t e = allow_smem<wkv6q_forward_kernel<M>>(Smem<M>::kBytes); \
        RWKV_REQUIRE(e == cudaSuccess, RWKVB200_ECUDA, "wkv6_forward: cudaFuncSetAttribute: %s", cudaGetErrorString(e));  \
        wkv6q_forward_kernel<M><<<grid, PNT, Smem<M>::kBytes, st>>>(T, H, maps, w, (const bf16*)u, s0, s0_kind, (bf16*)y, sT, \
                                                                ck, unsafe, flag_div);                                       \
    } while (0)
    switch (w_mode) {
        case 0: RWKV_GO(0); break;
        case 1: RWKV_GO(1); break;
        case 2: RWKV_GO(2); break;
        case 3: RWKV_GO(3); break;
        default: RWKV_GO(4); break;
    }
#undef RWKV_GO
    return check_launch("wkv6_forward(tcgen05, 32-token chunks, three stages)");
}

int wkv6_l32_error(int clear) {
    int h = 0;
    if (clear) return cudaMemcpyToSymbol(v6q::g_v6q_error, &h, sizeof(int)) == cudaSuccess ? 0 : -1;
    if (cudaMemcpyFromSymbol(&h, v6q::g_v6q_error, sizeof(int)) != cudaSuccess) return -1;
    return h;
}

}  // namespace rwkvb200
