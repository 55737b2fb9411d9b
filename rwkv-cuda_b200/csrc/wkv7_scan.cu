// RWKV-7 training, head size 64, bf16, for launches with few (batch, head) units: the chunks of a sequence are worked on at
// the same time, and only a short chain of products walks them in order.
//
// With the chunk algebra of wkv7_l32.cuh (scaled operands A~, R~, B~, K~, V, matrices U, T = (I - U_ab)^-1, chunk decay We)
// the end state of a chunk and its outputs are affine in its start state S (64 x 64, [value][key]):
//   S_end = (S + S Delta + G) diag(We)      Delta = A~^T T B~                    G  = V (U_ak T B~ + K~)
//   Y     = S Yop + Y0                      Yop   = R~^T + A~^T T U_br            Y0 = V (U_ak T U_br + U_kr)
// and, with Ew = E diag(We), the adjoint of the start state follows from the same two operators:
//   E_start = Ew + Ew Delta^T + dY Yop^T
// So: (1) one block per chunk makes Delta, Yop, G, Y0 (nothing of it depends on the state); (2) one block per unit walks the
// chunks with two products each, S in fp32 registers and, rounded to TF32, in tensor memory; (3) backward: one block per unit
// walks the adjoint the same way and leaves it at the end of every chunk; (4) wkv7_l32_bwd.cu runs with one block per chunk.
// The products of the chain are read as TF32 like every other operand; S, E and all sums stay fp32 (errors against fp64 as in the
// chunk-by-chunk kernels: sT 2.2e-4, ds0 2.1e-4).
//
// Measured on a B200, B2 T1040 H12 (24 units, 792 chunks): operators 19 us, chain 27 us (0.7 us per chunk against 2 us), adjoint
// chain 26 us (against 4.5 us per chunk), gradients 35 us; forward + backward 219 -> 113 us.  The chain of a chunk is one 64x64x64
// product and its way through registers; 16 stores of the state per thread beside it made it 1.0 us (see send_rows), y written
// by the same warps as long again.
//
// Record of a chunk, A (kept for the backward): Delta and Yop as the swizzled shared-memory images that the products read, We;
// B (dropped after the forward): G and Y0 in the order of the threads that add them.  Bulk copies bring records in whole.
#include <algorithm>
#include "wkv7_l32.cuh"
#include "wkv7_dispatch.cuh"

namespace rwkvb200 {
namespace v7s {

using namespace v7x;

constexpr int kRecA = ARR64 + HALF64 + 256;    // Delta [64][64], Yop [64 keys][32 tokens], We [64]
constexpr int kRecB = ARR64 + HALF64;          // G, Y0

__device__ int g_v7s_error = 0;

// Operand words hold the value plus half a unit of the last TF32 place (the tensor core drops the rest): this is the value itself.
__device__ __forceinline__ float unrounded(const unsigned char* p) { return __uint_as_float(*reinterpret_cast<const uint32_t*>(p) - 0x1000u); }
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_init_count(uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
// state rows -> tensor memory as an operand: rounded to TF32 here, because the tensor core truncates (S itself stays in registers)
__device__ __forceinline__ void put_operand(uint32_t taddr, const float (&x)[8][4]) {
    float q[8][4];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) q[nt][e] = tf32rf(x[nt][e]);
    tmem_st_tiles<8>(taddr, q);
    tmem_wait_st();
}
// ---- (1) the operators of a chunk ------------------------------------------------------------------------------
// Blocks walk over the chunks of all units (two blocks per SM); the tiles of a block's next chunk are on their way while it
// works on this one.
struct OpsSmem {
    static constexpr int kAR = 0, kBK = kAR + ARR64, kV = kBK + ARR64, kUak = kV + ARR32;
    static constexpr int kUbr = kUak + HALF32, kUkr = kUbr + HALF32, kD0 = kUkr + HALF32, kN1 = kD0 + HALF32;
    static constexpr int kRaw = kN1 + HALF32;               // six [32 tokens][64 channels] bf16 tiles
    static constexpr int kUab = kRaw + 6 * 4096;            // plain [32][UPITCH]
    static constexpr int kWe = kUab + 32 * UPITCH * 4, kHs = kWe + 256, kBar = kHs + 1024;
    static constexpr int kBytes = kBar + 64 + 1024;
};
static_assert(OpsSmem::kBytes <= 115712, "two blocks per SM");

__global__ void __launch_bounds__(128, 2) wkv7_ops_kernel(int T, int H, int nch, int total, const __grid_constant__ TileMaps<6> maps, unsigned char* __restrict__ recA,
                                                          unsigned char* __restrict__ recB) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    unsigned char *AR = smem + OpsSmem::kAR, *BK = smem + OpsSmem::kBK, *Vs = smem + OpsSmem::kV, *D0 = smem + OpsSmem::kD0, *N1 = smem + OpsSmem::kN1;
    unsigned char *Uak = smem + OpsSmem::kUak, *Ubr = smem + OpsSmem::kUbr, *Ukr = smem + OpsSmem::kUkr, *Raw = smem + OpsSmem::kRaw;
    float *Uab = reinterpret_cast<float*>(smem + OpsSmem::kUab), *We = reinterpret_cast<float*>(smem + OpsSmem::kWe), *Hs = reinterpret_cast<float*>(smem + OpsSmem::kHs);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + OpsSmem::kBar);   // tiles landed, U done, outputs done, the chain's own
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 4);

    const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int row0 = warp * 16;
    auto request = [&](int rec) {   // one thread: the six tiles of a chunk
        const int unit = rec / nch, c = rec - unit * nch, bb = unit / H, hh = unit - bb * H;
        mbar_expect_bytes(bar, 6 * 4096);
#pragma unroll
        for (int x = 0; x < 6; ++x) tma_tile_load(Raw + x * 4096, &maps.m[x], hh * 64, bb * T + c * LC, bar);
    };

    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) mbar_init(bar + i);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        request(blockIdx.x);
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(smem_u32(tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (int i = tid; i < 2 * HALF32 / 4; i += 128) reinterpret_cast<float*>(D0)[i] = 0.f;   // D0 and N1: the blocks never written stay zero
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem_slot[0], 0);
    // U, then G | Z = V U_ak, R, then Y0 | A~^T T | V U_ak T | R of the other chain, then Yop | Delta
    const uint32_t tmG = tm, tmZ = tm + 64, tmS1 = tm + 96, tmS2 = tm + 128, tmR = tm + 160, tmD = tm + 192;
    const uint32_t lane_off = (uint32_t)(warp * 32) << 16, lead = elect_one();
    const uint32_t arA = smem_u32(AR), bkA = smem_u32(BK), vA = smem_u32(Vs), uakA = smem_u32(Uak), ubrA = smem_u32(Ubr), ukrA = smem_u32(Ukr);
    const uint32_t d0A = smem_u32(D0), n1A = smem_u32(N1);
    ChainSync cs{bar + 3, 0, 0};   // used by warp 0 only
    int fail = 0;
    uint32_t par = 0;
    bool pending = true;           // tiles on their way that nobody has waited for

    for (int rec = blockIdx.x; rec < total; rec += gridDim.x, par ^= 1) {
        const int unit = rec / nch, valid = min(LC, T - (rec - unit * nch) * LC);
        if (!mbar_wait(bar, par)) fail = 1;
        pending = false;
        RawChunk<6, 8> raw;
        take_chunk<6, 8>(raw, Raw, valid, warp, lane);
        prepare_operands<6, 8, 4>(raw, AR, BK, Vs, HALF32, nullptr, 0, We, Hs, nullptr, warp, lane);
        proxy_fence();
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        pending = rec + (int)gridDim.x < total;
        if (pending && tid == 0) request(rec + gridDim.x);   // every thread has taken its part of the tiles
        if (warp == 0) {
            issue_u(tmG, arA, bkA, lead);
            mma_commit(bar + 1, lead);
        }
        if (!mbar_wait(bar + 1, par)) fail = 2;
        tc_fence_after();
        {
            float u[8][4];
            tmem_ld_tiles<8>(u, tmG + lane_off);
            tmem_wait_ld();
            scatter_u(u, warp, lane, Uab, N1, Uak, Ubr, Ukr);
        }
        tc_fence_before();
        __syncthreads();
        if (warp < 2) tri_inverse16<UPITCH>(Uab + 16 * warp * (UPITCH + 1), D0, 16 * warp, lane);
        proxy_fence();
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        if (warp == 0) {
            const uint32_t id32s = idesc64(32, 1, 1), id32t = idesc64(32, 0, 1), id64s = idesc64(64, 1, 1), id64t = idesc64(64, 0, 1);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) mma_ss(tmZ, desc_mn(vA, ks * 8, HALF32), desc_mn(uakA, ks * 8, HALF32), id32s, ks > 0, lead);    // Z = V U_ak
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) mma_ss(tmS1, desc_mn(arA, ks * 8, HALF64), desc_mn(d0A, ks * 8, HALF32), id32s, ks > 0, lead);   // A~^T D0
            cs.commit(lead);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) mma_ss(tmG, desc_mn(vA, ks * 8, HALF32), desc_mn(bkA + 32 * 128, ks * 8, HALF64), id64s, ks > 0, lead);   // G = V K~
            cs.wait();
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) mma_ts(tmS2, tmZ + ks * 8, desc_mn(d0A, ks * 8, HALF32), id32t, ks > 0, lead);   // Z D0
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) mma_ts(tmR, tmS1 + ks * 8, desc_mn(n1A, ks * 8, HALF32), id32t, ks > 0, lead);   // (A~^T D0) N1
            cs.sync(lead);
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) mma_ts(tmZ, tmS2 + ks * 8, desc_mn(n1A, ks * 8, HALF32), id32t, ks > 0, lead);   // (Z D0) N1
#pragma unroll
            for (int ks = 2; ks < 4; ++ks) mma_ts(tmS1, tmR + ks * 8, desc_mn(d0A, ks * 8, HALF32), id32t, 1, lead);        // A~^T T
            cs.sync(lead);
#pragma unroll
            for (int ks = 2; ks < 4; ++ks) mma_ts(tmS2, tmZ + ks * 8, desc_mn(d0A, ks * 8, HALF32), id32t, 1, lead);        // V U_ak T
            cs.commit(lead);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) mma_ts(tmD, tmS1 + ks * 8, desc_mn(bkA, ks * 8, HALF64), id64t, ks > 0, lead);   // Delta
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) mma_ts(tmR, tmS1 + ks * 8, desc_mn(ubrA, ks * 8, HALF32), id32t, ks > 0, lead);  // Yop (R~^T is added below)
            cs.wait();
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) mma_ts(tmG, tmS2 + ks * 8, desc_mn(bkA, ks * 8, HALF64), id64t, 1, lead);        // G += V U_ak T B~
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) mma_ss(tmZ, desc_mn(vA, ks * 8, HALF32), desc_mn(ukrA, ks * 8, HALF32), id32s, ks > 0, lead);    // Y0 = V U_kr
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) mma_ts(tmZ, tmS2 + ks * 8, desc_mn(ubrA, ks * 8, HALF32), id32t, 1, lead);       //    + V U_ak T U_br
            mma_commit(bar + 2, lead);
            if (cs.fail) fail = 3;
        }
        if (!mbar_wait(bar + 2, par)) fail = 4;
        tc_fence_after();
        {
            unsigned char* A = recA + (i64)rec * kRecA;
            float4* Bo = reinterpret_cast<float4*>(recB + (i64)rec * kRecB);
            float d[8][4];
            tmem_ld_tiles<8>(d, tmD + lane_off);
            tmem_wait_ld();
#pragma unroll
            for (int nt = 0; nt < 8; ++nt)
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    *reinterpret_cast<float2*>(A + sw(row0 + g + 8 * h, nt * 8 + 2 * t, HALF64)) = make_float2(tf32rf(d[nt][2 * h]), tf32rf(d[nt][2 * h + 1]));
            float y[4][4];
            tmem_ld_tiles<4>(y, tmR + lane_off);
            tmem_wait_ld();
#pragma unroll
            for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int j = row0 + g + 8 * h, tt = nt * 8 + 2 * t;
                    const float r0 = unrounded(AR + sw(32 + tt, j, HALF64)), r1 = unrounded(AR + sw(33 + tt, j, HALF64));
                    *reinterpret_cast<float2*>(A + ARR64 + sw32(j, tt)) = make_float2(tf32rf(y[nt][2 * h] + r0), tf32rf(y[nt][2 * h + 1] + r1));
                }
            if (tid < 64) reinterpret_cast<float*>(A + ARR64 + HALF64)[tid] = We[tid];
            tmem_ld_tiles<8>(d, tmG + lane_off);
            tmem_ld_tiles<4>(y, tmZ + lane_off);
            tmem_wait_ld();
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) Bo[nt * 128 + tid] = make_float4(d[nt][0], d[nt][1], d[nt][2], d[nt][3]);
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) Bo[8 * 128 + nt * 128 + tid] = make_float4(y[nt][0], y[nt][1], y[nt][2], y[nt][3]);
        }
        if (fail) reinterpret_cast<float*>(recA + (i64)rec * kRecA)[0] = __int_as_float(0x7fc00000);   // the chain carries it into the outputs
        tc_fence_before();
        if (__syncthreads_or(fail)) { par ^= 1; break; }   // (and: the operand arrays may be written again)
        tc_fence_after();
    }
    if (pending && fail) mbar_wait(bar, par);   // leaving early: the requested tiles must have landed before the block may end
    if (fail) atomicMax(&g_v7s_error, fail);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tm) : "memory");
}

// ---- (2), (3) the chain ------------------------------------------------------------------------------------------
constexpr int NSTG = 3;   // records in flight

struct ChainSmem {
    static constexpr int kStage = ARR64 + HALF64 + ARR64 + HALF64 + 1024;   // Delta, Yop, then G and Y0 (backward: dY as operand, its raw tile), We
    static constexpr int kWe = ARR64 + HALF64 + ARR64 + HALF64;
    static constexpr int kY = NSTG * kStage;                                // bf16 [32][72]
    static constexpr int kOut = (kY + 32 * 72 * 2 + 1023) / 1024 * 1024;    // two images of S (or E) on their way out
    static constexpr int kBar = kOut + 2 * ARR64;
    static constexpr int kBytes = kBar + 256 + 1024;
};
static_assert(ChainSmem::kStage % 1024 == 0 && ChainSmem::kBytes <= 232448, "layout");
enum { kFull = 0, kEmpty = kFull + NSTG, kOper = kEmpty + NSTG, kState = kOper + NSTG, kProdD, kProdY, kYTaken = kProdY + 2, kNBarC = kYTaken + 2 };

// Arrival of a warp (after what its lanes have done): one lane arrives, 32 arrivals on one word would queue up.
__device__ __forceinline__ void warp_arrive(uint64_t* bar, int lane) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}

// Forward: warps 0-3 carry S in fp32 registers (16 value rows each) and write the states and sT; warps 4-7 write y; warp 8 issues
// the products; warp 9 asks for the records.  A waiter may be one phase of an mbarrier behind, not two: the Y product and its
// release have an mbarrier for even and one for odd chunks.  grid (H, B).  states: S at the start of
// every chunk, as images of the operand array that the backward makes of it.
__global__ void __launch_bounds__(320, 1) wkv7_chain_forward_kernel(int T, int H, int nch, const float* __restrict__ s0_, const unsigned char* __restrict__ recA,
                                                                    const unsigned char* __restrict__ recB, bf16* __restrict__ y_,
                                                                    float* __restrict__ sT_, float* __restrict__ states) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    bf16* ystage = reinterpret_cast<bf16*>(smem + ChainSmem::kY);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + ChainSmem::kBar);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + kNBarC);
    volatile int* abort_word = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* gabort = abort_word + 1;   // the value on which warps 0-3 decide together
    const int hh = blockIdx.x, bb = blockIdx.y, unit = bb * H + hh, C = H * 64;
    const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < kNBarC; ++i) mbar_init_count(bar + i, i == kState || i == kYTaken || i == kYTaken + 1 ? 4 : i >= kEmpty && i < kEmpty + NSTG ? 8 : 1);
        *abort_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(smem_u32(tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem_slot[0], 0);   // S of even and odd chunks | S Delta | Y of even and odd chunks
    const uint32_t tmD = tm + 128, tmY = tm + 192;
    int fail = 0;

    if (warp == 9) {
        if (lane == 0) {
            int c = 0;
            for (; c < nch; ++c) {
                const int st = c % NSTG, n = c / NSTG;
                if (n > 0 && !mbar_wait(bar + kEmpty + st, (n - 1) & 1)) { fail = 1; break; }
                if (*abort_word) break;
                unsigned char* s = smem + st * ChainSmem::kStage;
                const i64 rec = (i64)unit * nch + c;
                mbar_expect_bytes(bar + kFull + st, kRecA + kRecB);
                bulk_load(s, recA + rec * kRecA, ARR64 + HALF64, bar + kFull + st);
                bulk_load(s + ChainSmem::kWe, recA + rec * kRecA + ARR64 + HALF64, 256, bar + kFull + st);
                bulk_load(s + ARR64 + HALF64, recB + rec * kRecB, kRecB, bar + kFull + st);
            }
            if (fail) atomicMax(const_cast<int*>(abort_word), fail);
            if (*abort_word)   // leaving early: the copies in flight must have landed before the block may end
                for (int cc = max(0, c - NSTG); cc < c; ++cc) mbar_wait(bar + kFull + cc % NSTG, (cc / NSTG) & 1);
        }
    } else if (warp == 8) {
        const uint32_t lead = elect_one(), idD = idesc64(64, 0, 1), idY = idesc64(32, 0, 1);
        for (int c = 0; c < nch; ++c) {
            const int st = c % NSTG;
            if (!mbar_wait(bar + kFull + st, (c / NSTG) & 1)) fail = 2;
            if (!mbar_wait(bar + kState, c & 1)) fail = 3;
            if (__any_sync(0xffffffffu, fail)) break;
            tc_fence_after();
            const uint32_t dA = smem_u32(smem + st * ChainSmem::kStage), yA = dA + ARR64, tmS = tm + (c & 1) * 64;
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) mma_ts(tmD, tmS + ks * 8, desc_mn(dA, ks * 8, HALF64), idD, ks > 0, lead);   // S Delta
            mma_commit(bar + kProdD, lead);
            if (c > 1 && !mbar_wait(bar + kYTaken + (c & 1), ((c >> 1) - 1) & 1)) fail = 7;   // the Y of two chunks ago has been read
            if (__any_sync(0xffffffffu, fail)) break;
            tc_fence_after();
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) mma_ts(tmY + (c & 1) * 32, tmS + ks * 8, desc_mn(yA, ks * 8, HALF64), idY, ks > 0, lead);   // S Yop
            mma_commit(bar + kProdY + (c & 1), lead);
        }
        if (fail && lane == 0) atomicMax(const_cast<int*>(abort_word), fail);
    } else if (warp >= 4) {
        // y: the product and Y0, out as rows of bf16
        const int quarter = warp & 3, gtid = tid & 127, row0 = quarter * 16;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        const i64 tok0 = (i64)bb * T * C + hh * 64;
        for (int c = 0; c < nch; ++c) {
            const int st = c % NSTG, valid = min(LC, T - c * LC);
            const float4* Y0 = reinterpret_cast<const float4*>(smem + st * ChainSmem::kStage + 2 * ARR64 + HALF64);
            if (!mbar_wait(bar + kFull + st, (c / NSTG) & 1)) fail = 8;
            if (!mbar_wait(bar + kProdY + (c & 1), (c >> 1) & 1)) fail = 6;
            tc_fence_after();
            float y[4][4];
            tmem_ld_tiles<4>(y, tmY + (c & 1) * 32 + lane_off);
            tmem_wait_ld();
            tc_fence_before();
            warp_arrive(bar + kYTaken + (c & 1), lane);
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                const float4 q = Y0[nt * 128 + gtid];
                const float add[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    ystage[(nt * 8 + 2 * t + (e & 1)) * 72 + row0 + g + ((e & 2) ? 8 : 0)] = __float2bfloat16_rn(y[nt][e] + add[e]);
            }
            warp_arrive(bar + kEmpty + st, lane);   // (the product has read the record: it is complete)
            if (fail) atomicMax(const_cast<int*>(abort_word), fail);
            if (gtid == 0) *gabort = *abort_word;
            group_sync(1, 128);
            const int stop = *gabort, tt = gtid >> 2, q = gtid & 3;
            if (tt < valid) {
                const uint4* sp = reinterpret_cast<const uint4*>(ystage + tt * 72 + q * 16);
                uint4* dp = reinterpret_cast<uint4*>(y_ + tok0 + (i64)(c * LC + tt) * C + q * 16);
                dp[0] = sp[0];
                dp[1] = sp[1];
            }
            if (stop) break;
            group_sync(2, 128);                     // the staging rows may be written again
        }
    } else {
        const uint32_t lane_off = (uint32_t)(warp * 32) << 16;
        const int row0 = warp * 16;
        const i64 sbase = (i64)unit * 4096;
        unsigned char* st_out = reinterpret_cast<unsigned char*>(states) + (i64)unit * nch * ARR64;
        auto put_state = [&](float* dst, const float (&S)[8][4]) {
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                *reinterpret_cast<float2*>(dst + (row0 + g) * 64 + nt * 8 + 2 * t) = make_float2(S[nt][0], S[nt][1]);
                *reinterpret_cast<float2*>(dst + (row0 + g + 8) * 64 + nt * 8 + 2 * t) = make_float2(S[nt][2], S[nt][3]);
            }
        };
        float S[8][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            float2 lo = make_float2(0.f, 0.f), hi = lo;
            if (s0_ != nullptr) {
                lo = *reinterpret_cast<const float2*>(s0_ + sbase + (row0 + g) * 64 + nt * 8 + 2 * t);
                hi = *reinterpret_cast<const float2*>(s0_ + sbase + (row0 + g + 8) * 64 + nt * 8 + 2 * t);
            }
            S[nt][0] = lo.x; S[nt][1] = lo.y; S[nt][2] = hi.x; S[nt][3] = hi.y;
        }
        put_operand(tm + lane_off, S);
        tc_fence_before();
        warp_arrive(bar + kState, lane);
        send_rows(smem + ChainSmem::kOut, 0, st_out, S, row0, lane);
        for (int c = 0; c < nch; ++c) {
            const int st = c % NSTG;
            const unsigned char* s = smem + st * ChainSmem::kStage;
            const float4 *G = reinterpret_cast<const float4*>(s + ARR64 + HALF64);
            const float* We = reinterpret_cast<const float*>(s + ChainSmem::kWe);
            if (!mbar_wait(bar + kFull + st, (c / NSTG) & 1)) fail = 4;
            // (S + G) diag(We) is ready before the product is
            float2 we[8];
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                const float4 q = G[nt * 128 + tid];
                we[nt] = *reinterpret_cast<const float2*>(We + nt * 8 + 2 * t);
                S[nt][0] = (S[nt][0] + q.x) * we[nt].x; S[nt][1] = (S[nt][1] + q.y) * we[nt].y;
                S[nt][2] = (S[nt][2] + q.z) * we[nt].x; S[nt][3] = (S[nt][3] + q.w) * we[nt].y;
            }
            if (!mbar_wait(bar + kProdD, c & 1)) fail = 5;
            tc_fence_after();
            {
                float d[8][4];
                tmem_ld_tiles<8>(d, tmD + lane_off);
                tmem_wait_ld();
#pragma unroll
                for (int nt = 0; nt < 8; ++nt) {
                    S[nt][0] = fmaf(d[nt][0], we[nt].x, S[nt][0]); S[nt][1] = fmaf(d[nt][1], we[nt].y, S[nt][1]);
                    S[nt][2] = fmaf(d[nt][2], we[nt].x, S[nt][2]); S[nt][3] = fmaf(d[nt][3], we[nt].y, S[nt][3]);
                }
            }
            if (c + 1 < nch) {
                put_operand(tm + ((c + 1) & 1) * 64 + lane_off, S);
                tc_fence_before();
                warp_arrive(bar + kState, lane);   // the next chunk's products may start
                send_rows(smem + ChainSmem::kOut, c + 1, st_out + (i64)(c + 1) * ARR64, S, row0, lane);
            } else if (sT_ != nullptr) {
                put_state(sT_ + sbase, S);
            }
            warp_arrive(bar + kEmpty + st, lane);
            if (__any_sync(0xffffffffu, fail)) break;
        }
        sent_all(lane);
        if (fail) atomicMax(const_cast<int*>(abort_word), fail);
    }
    tc_fence_before();
    __syncthreads();
    if (*abort_word && tid == 0) {
        atomicMax(&g_v7s_error, *abort_word);
        y_[(i64)bb * T * C + hh * 64] = __ushort_as_bfloat16((unsigned short)0x7fc0);
    }
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tm) : "memory");
}

// Backward: the same roles with E; warps 6 and 7 turn the tile of dY into an operand.  E at the end of every chunk is written to
// `adjoints` (images like the states), the adjoint of the initial state to ds0.
__global__ void __launch_bounds__(256, 1) wkv7_chain_backward_kernel(int T, int H, int nch, const float* __restrict__ dsT_,
                                                                     const __grid_constant__ CUtensorMap dymap, const unsigned char* __restrict__ recA,
                                                                     float* __restrict__ adjoints, float* __restrict__ ds0_) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + ChainSmem::kBar);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + kNBarC);
    volatile int* abort_word = reinterpret_cast<volatile int*>(tmem_slot + 1);
    constexpr int kOperand = ARR64 + HALF64, kTile = kOperand + ARR32;   // dY in a stage: operand [32][64], tile
    const int hh = blockIdx.x, bb = blockIdx.y, unit = bb * H + hh;
    const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < kNBarC; ++i)
            mbar_init_count(bar + i, i == kState || (i >= kEmpty && i < kEmpty + NSTG) ? 4 : i >= kOper && i < kOper + NSTG ? 2 : 1);
        *abort_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(smem_u32(tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem_slot[0], 0), tmD = tm + 64;   // Ew | products of even and odd steps
    int fail = 0;

    if (warp == 5) {
        if (lane == 0) {
            int n = 0;   // step n works on chunk nch - 1 - n
            for (; n < nch; ++n) {
                const int st = n % NSTG, k = n / NSTG, c = nch - 1 - n;
                if (k > 0 && !mbar_wait(bar + kEmpty + st, (k - 1) & 1)) { fail = 11; break; }
                if (*abort_word) break;
                unsigned char* s = smem + st * ChainSmem::kStage;
                const i64 rec = (i64)unit * nch + c;
                mbar_expect_bytes(bar + kFull + st, kRecA + 4096);
                bulk_load(s, recA + rec * kRecA, ARR64 + HALF64, bar + kFull + st);
                bulk_load(s + ChainSmem::kWe, recA + rec * kRecA + ARR64 + HALF64, 256, bar + kFull + st);
                tma_tile_load(s + kTile, &dymap, hh * 64, bb * T + c * LC, bar + kFull + st);
            }
            if (fail) atomicMax(const_cast<int*>(abort_word), fail);
            if (*abort_word)
                for (int m = max(0, n - NSTG); m < n; ++m) mbar_wait(bar + kFull + m % NSTG, (m / NSTG) & 1);
        }
    } else if (warp >= 6) {
        for (int n = 0; n < nch; ++n) {
            const int st = n % NSTG, valid = min(LC, T - (nch - 1 - n) * LC);
            if (!mbar_wait(bar + kFull + st, (n / NSTG) & 1)) fail = 12;
            if (__any_sync(0xffffffffu, fail)) break;
            unsigned char* s = smem + st * ChainSmem::kStage;
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                const int tt = 16 * (warp - 6) + q;
                const uint32_t x = tt < valid ? *reinterpret_cast<const uint32_t*>(s + kTile + tt * 128 + 4 * lane) : 0u;
                *reinterpret_cast<float2*>(s + kOperand + sw(tt, 2 * lane, HALF32)) = bf16x2_to_f2(x);
            }
            proxy_fence();
            warp_arrive(bar + kOper + st, lane);
        }
        if (fail && lane == 0) atomicMax(const_cast<int*>(abort_word), fail);
    } else if (warp == 4) {
        const uint32_t lead = elect_one(), idY = idesc64(64, 1, 0), idE = idesc64(64, 0, 0);
        for (int n = 0; n <= nch; ++n) {
            if (n > 0) {   // Ew Delta^T of step n - 1
                if (!mbar_wait(bar + kState, (n - 1) & 1)) fail = 13;
                if (__any_sync(0xffffffffu, fail)) break;
                tc_fence_after();
                const uint32_t dA = smem_u32(smem + ((n - 1) % NSTG) * ChainSmem::kStage);
#pragma unroll
                for (int ks = 0; ks < 8; ++ks) mma_ts(tmD + ((n - 1) & 1) * 64, tm + ks * 8, desc_k(dA, 0, ks * 8, HALF64), idE, 1, lead);
                mma_commit(bar + kProdD, lead);
            }
            if (n == nch) break;
            const int st = n % NSTG;   // dY Yop^T of step n needs no state: it is under way before the state arrives
            if (!mbar_wait(bar + kOper + st, (n / NSTG) & 1)) fail = 14;
            if (__any_sync(0xffffffffu, fail)) break;
            tc_fence_after();
            const uint32_t yA = smem_u32(smem + st * ChainSmem::kStage + ARR64), oA = smem_u32(smem + st * ChainSmem::kStage + kOperand);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) mma_ss(tmD + (n & 1) * 64, desc_mn(oA, ks * 8, HALF32), desc_k(yA, 0, ks * 8, HALF64), idY, ks > 0, lead);
        }
        if (fail && lane == 0) atomicMax(const_cast<int*>(abort_word), fail);
    } else {
        const uint32_t lane_off = (uint32_t)(warp * 32) << 16;
        const int row0 = warp * 16;
        const i64 sbase = (i64)unit * 4096;
        auto put = [&](float* dst, const float (&x)[8][4]) {
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                *reinterpret_cast<float2*>(dst + (row0 + g) * 64 + nt * 8 + 2 * t) = make_float2(x[nt][0], x[nt][1]);
                *reinterpret_cast<float2*>(dst + (row0 + g + 8) * 64 + nt * 8 + 2 * t) = make_float2(x[nt][2], x[nt][3]);
            }
        };
        float E[8][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            float2 lo = make_float2(0.f, 0.f), hi = lo;
            if (dsT_ != nullptr) {
                lo = *reinterpret_cast<const float2*>(dsT_ + sbase + (row0 + g) * 64 + nt * 8 + 2 * t);
                hi = *reinterpret_cast<const float2*>(dsT_ + sbase + (row0 + g + 8) * 64 + nt * 8 + 2 * t);
            }
            E[nt][0] = lo.x; E[nt][1] = lo.y; E[nt][2] = hi.x; E[nt][3] = hi.y;
        }
        for (int n = 0; n < nch; ++n) {
            const int st = n % NSTG, c = nch - 1 - n;
            const float* We = reinterpret_cast<const float*>(smem + st * ChainSmem::kStage + ChainSmem::kWe);
            if (!mbar_wait(bar + kFull + st, (n / NSTG) & 1)) fail = 15;
            float Ew[8][4];
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                const float2 we = *reinterpret_cast<const float2*>(We + nt * 8 + 2 * t);
                Ew[nt][0] = E[nt][0] * we.x; Ew[nt][1] = E[nt][1] * we.y; Ew[nt][2] = E[nt][2] * we.x; Ew[nt][3] = E[nt][3] * we.y;
            }
            put_operand(tm + lane_off, Ew);
            tc_fence_before();
            warp_arrive(bar + kState, lane);
            send_rows(smem + ChainSmem::kOut, n, reinterpret_cast<unsigned char*>(adjoints) + ((i64)unit * nch + c) * ARR64, E, row0, lane);
            if (!mbar_wait(bar + kProdD, n & 1)) fail = 16;
            tc_fence_after();
            tmem_ld_tiles<8>(E, tmD + (n & 1) * 64 + lane_off);
            tmem_wait_ld();
            tc_fence_before();
#pragma unroll
            for (int nt = 0; nt < 8; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) E[nt][e] += Ew[nt][e];
            warp_arrive(bar + kEmpty + st, lane);
            if (__any_sync(0xffffffffu, fail)) break;
        }
        sent_all(lane);
        if (fail) atomicMax(const_cast<int*>(abort_word), fail);
        if (ds0_ != nullptr) put(ds0_ + sbase, E);
    }
    tc_fence_before();
    __syncthreads();
    if (*abort_word && tid == 0) {
        atomicMax(&g_v7s_error, *abort_word);
        adjoints[(i64)unit * nch * 4096] = __int_as_float(0x7fc00000);
    }
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tm) : "memory");
}

}  // namespace v7s

size_t wkv7_scan_saved_bytes(int B, int T, int H) { return (size_t)B * H * ((T + 31) / 32) * (v7s::kRecA + 64 * 64 * sizeof(float)); }
size_t wkv7_scan_work_bytes(int B, int T, int H, bool backward) {
    return (size_t)B * H * ((T + 31) / 32) * (backward ? 64 * 64 * sizeof(float) : (size_t)v7s::kRecB);
}

int wkv7_scan_forward(int B, int T, int H, const float* s0, const void* r, const void* w, const void* k, const void* v, const void* a,
                      const void* b, void* y, float* sT, void* saved, void* work, cudaStream_t st) {
    using namespace v7s;
    const int nch = (T + 31) / 32;
    TileMaps<6> maps;
    const void* in[6] = {r, w, k, v, a, b};
    make_tile_maps<6>(maps, in, B, T, H);
    if (!maps.valid) return 1;
    cudaError_t e = allow_smem<wkv7_ops_kernel>(OpsSmem::kBytes);
    if (e == cudaSuccess) e = allow_smem<wkv7_chain_forward_kernel>(ChainSmem::kBytes);
    RWKV_REQUIRE(e == cudaSuccess, RWKVB200_ECUDA, "wkv7_train_forward: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    float* states = static_cast<float*>(saved);
    unsigned char* recA = static_cast<unsigned char*>(saved) + (size_t)B * H * nch * 64 * 64 * sizeof(float);
    const long long total = (long long)B * H * nch;
    RWKV_REQUIRE(total < (1ll << 31), RWKVB200_EINVAL, "wkv7_train_forward: too many chunks");
    wkv7_ops_kernel<<<(int)std::min<long long>(total, 2 * std::max(1, sm_count())), 128, OpsSmem::kBytes, st>>>(T, H, nch, (int)total, maps, recA, static_cast<unsigned char*>(work));
    wkv7_chain_forward_kernel<<<dim3(H, B), 320, ChainSmem::kBytes, st>>>(T, H, nch, s0, recA, static_cast<unsigned char*>(work), (bf16*)y, sT, states);
    return check_launch("wkv7_train_forward(chunks in parallel)");
}

int wkv7_scan_backward(int B, int T, int H, const void* r, const void* w, const void* k, const void* v, const void* a, const void* b,
                       const void* dy, const float* dsT, const void* saved, void* work, float* ds0, void* dr, void* dw, void* dk, void* dv,
                       void* da, void* db, cudaStream_t st) {
    using namespace v7s;
    const int nch = (T + 31) / 32;
    CUtensorMap dymap;
    RWKV_REQUIRE(wkv7_make_tile_map(&dymap, dy, (unsigned long long)B * T, (unsigned long long)H * 64), RWKVB200_EUNSUPPORTED,
                 "wkv7_train_backward: no tensor map for dy");
    const cudaError_t e = allow_smem<wkv7_chain_backward_kernel>(ChainSmem::kBytes);
    RWKV_REQUIRE(e == cudaSuccess, RWKVB200_ECUDA, "wkv7_train_backward: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    const float* states = static_cast<const float*>(saved);
    const unsigned char* recA = static_cast<const unsigned char*>(saved) + (size_t)B * H * nch * 64 * 64 * sizeof(float);
    float* adjoints = static_cast<float*>(work);
    wkv7_chain_backward_kernel<<<dim3(H, B), 256, ChainSmem::kBytes, st>>>(T, H, nch, dsT, dymap, recA, adjoints, ds0);
    if (int rc = check_launch("wkv7_train_backward(chain)")) return rc;
    return wkv7_l32_backward_chunks(B, T, H, r, w, k, v, a, b, dy, adjoints, states, dr, dw, dk, dv, da, db, st);
}

int wkv7_scan_error(int clear) {
    int h = 0;
    if (clear) return cudaMemcpyToSymbol(v7s::g_v7s_error, &h, sizeof(int)) == cudaSuccess ? 0 : -1;
    if (cudaMemcpyFromSymbol(&h, v7s::g_v7s_error, sizeof(int)) != cudaSuccess) return -1;
    return h;
}

}  // namespace rwkvb200
