// Matrix forms of the kernels that work on the time segments of a sequence at the same time (wkv5_seg.cu, wkv6_seg.cu): head
// size 64, segments of 32 tokens, fp32 or bf16 activations, products of 24-bit operands and fp32 states.
//
// Inside a segment the recurrence is a set of small products (S: state before the segment, D: adjoint after it, both [key j]
// [value i]; L_t: sum of log decays up to token t; m: the middle of the segment, where the scaled vectors are anchored so that
// neither side of a product runs out of fp32's range):
//   r~_t = r_t exp(L_{t-1} - L_m)    k~_s = k_s exp(L_m - L_s)    S' = exp(L_m) S    D' = exp(L_end - L_m) D
//   A[s,t] = k~_s.r~_t (s < t), A[t,t] = sum_j r_t u k_t      G[s,t] = v_s.gy_t (s < t), gamma_t = v_t.gy_t
//   y  = R~ S' + A^T V
//   gv = K~ D' + A gY      dk~ = V D'^T + G R~      dr~ = gY S'^T + G^T K~
//   gk_s = dk~_s exp(L_m - L_s) + gamma_s u r_s     gr_t = dr~_t exp(L_{t-1} - L_m) + gamma_t u k_t
// and with P_t = r~_t dr~_t, Q_s = k~_s dk~_s (elementwise, without the u terms) and A_end = sum_i D S_end
//   dL/dlog d_t = A_end - sum_{tau > t} (Q_tau - P_tau) - Q_t      A_end = sum_i D' S' + sum_s k~_s (V D'^T)_s
// A static decay has the sum of these over the tokens, where terms that no decay acts on stand many times and cancel (error of gw at
// decays of 0.7 per token 1.0e-6 of its norm, token by token 2.9e-7); so in fp32 every term times the number of decays in it
// (n: tokens of the segment, t from 0), 2.0e-7:
//   dL/dlog d = n sum_i D' S' + sum_s (n-1-s) k~_s (V D'^T)_s + sum_t t r~_t (gY S'^T)_t + sum_t r~_t sum_{s<t} (t-1-s) G[s,t] k~_s
//
// Precision: the products run on mma.sync with bf16 operands, every fp32 operand as the sum of three bf16 numbers (24 bits: the
// split is exact) and all partial products down to 2^-16 of the largest taken: 3 where the other side is a bf16 tensor as it
// came, else 6.  What is left out is below 2^-25 of a product.  The split keeps its 24 bits as long as the last part is not below 2^-133: values
// from 2^-109 on, times what scales them (kRange, kStaticRange).  The tensor core cuts its sums off instead of rounding them.  Where a
// result is fp32 every group of products is summed from zero and added with rounding, and so is a segment's part of a state; y and
// gradients in bf16 accumulate on the tensor core over one segment (5.9e-7 of the norm against 4.4e-7, where the rounding to bf16 makes 1.66e-3:
// results equal to four digits at all decays, and 497 us instead of 526 for B8 T1000 H32).
// Why mma.sync and not tcgen05: these kernels are a block per segment with every accumulator and both states in registers,
// three to five blocks per SM; the operands are split where they are used, and at 8 clocks per instruction and scheduler the tensor pipe
// needs about as long as the arithmetic around it.
// B8 T1000 H32 bf16: backward kernel 251 us (314 with a channel order in which a lane has two neighbours and not four, rows of
// exponents 64 floats apart, the token matrices as fp32, a test of the alignment per load, bf16 parts unpacked before they are
// subtracted and states read where they are used), y 105 us (110 with four blocks per SM and 125 registers a thread instead of five
// and 96).  3700 instructions a warp, 324 of them mma: issue slots and the latency of 16 warps per SM (128 registers a thread) bound
// it, the tensor pipe is busy 30 % of the time.
// A segment whose decays leave the range (more than kRange between its middle and an end), that holds values that are not
// finite (a masked product would spread them over tokens before) or whose results are not (a state that is not finite; scaled operands
// whose product overflows although the result would not) is flagged and left to the token-by-token kernels.  Static decays are looked at where
// the states are made, decays per token there too with few units (the walk took 64 -> 72 us with it), else at the first barrier here.
#pragma once
#include "seg_tiles.cuh"

namespace rwkvb200 {
namespace {

// log2 of the largest decay between the middle of a segment and an end of it.  A value scaled by 2^-48 and split in three keeps its 24 bits
// down to 2^-133, so from 4e-19 on, and 12 of them from 9e-23 on; the logarithms' rounding makes 2e-6.  (With 86 gradients of 1e-14
// kept three bits and the decay gradient of a channel just inside had an error of 4.6e-3 at its worst element, 3.9e-3 being its rounding
// to bf16; with 60 it was 3.97e-3.  With 32, inputs of w around -1 +- 1 flag so many segments that B8 T1000 H32 takes 1140 us, 620 with 48.)
constexpr float kRange = 48.f;
// log2 of the largest decay of one token that is the same for all tokens: a factor of 2.  (Of a token and not up to the middle, which
// let a short last segment have more: at T 34 a factor of 256.)  Errors of y in fp32, products / token by token, of the norm: w from -6 to -1
// 1.8e-7 / 5.2e-7, -1.2 to -1 1.15e-7 / 1.11e-7, -1 to -0.4 1.12e-7 / 9.4e-8 where all channels of a head are that fast; slower ones decide beside them.
constexpr float kStaticRange = 1.f;
constexpr float kLog2e = 1.4426950408889634f;
constexpr int kImg = kSeg * 128;               // bytes of one bf16 image [32 tokens][64 channels]
constexpr int kTiles = 3 * 512;                // bytes of one bf16 image of a triangular token x token matrix: its 16 x 16 tiles
constexpr int kRld = 80;                       // floats of a row of 64 channels: 16-byte reads of two rows hit every bank once

// ---- bf16 images: rows of 128 bytes, their 16-byte pieces XOR-ed with the row ------------------------------------------------
// The channels of each group of 16 stand in the order 0 1 4 5 8 9 12 13 2 3 6 7 10 11 14 15.  A lane's four k of a product over channels
// and the four columns that it gets in two tiles are then neighbours, channels 4 q .. 4 q + 3: states, inputs and outputs move in
// pieces of four (in the plain order of two: the backward kernel's load/store pipe was busy 70 % of the time with lines
// that were touched twice, and B8 T1000 H32 took 544 us forward + backward instead of 510).
// Row (or column) g of a tile is channel at16(g), of the tile beside it at16(g) + 2.
__device__ __forceinline__ int at16(int g) { return 4 * (g >> 1) + (g & 1); }
__device__ __forceinline__ uint32_t img_at(int row, int piece) { return row * 128 + ((piece ^ (row & 7)) << 4); }
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// Fragments of mma.m16n8k16 by ldmatrix.  The place that a lane points at: (r0, c0) = first row, first 16-byte piece.
//   frag_rows: A[m][k] from rows m, B[k][n] from rows k (transposed);  frag_cols: A from rows k (transposed), B from rows n
// an x4 load is one A fragment, or the B fragments of two neighbouring n-tiles.
__device__ __forceinline__ uint32_t frag_rows(int r0, int c0, int lane) { return img_at(r0 + (lane & 15), c0 + (lane >> 4)); }
__device__ __forceinline__ uint32_t frag_cols(int r0, int c0, int lane) { return img_at(r0 + (lane & 7) + ((lane >> 4) << 3), c0 + ((lane >> 3) & 1)); }
__device__ __forceinline__ void ldsm(uint32_t (&f)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(f[0]), "=r"(f[1]), "=r"(f[2]), "=r"(f[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_t(uint32_t (&f)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(f[0]), "=r"(f[1]), "=r"(f[2]), "=r"(f[3]) : "r"(addr));
}
template <int NS, int STEP = kImg>
__device__ __forceinline__ void ldsm(uint32_t (&f)[NS][4], uint32_t addr) {
#pragma unroll
    for (int s = 0; s < NS; ++s) ldsm(f[s], addr + s * STEP);
}
template <int NS, int STEP = kImg>
__device__ __forceinline__ void ldsm_t(uint32_t (&f)[NS][4], uint32_t addr) {
#pragma unroll
    for (int s = 0; s < NS; ++s) ldsm_t(f[s], addr + s * STEP);
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// c[mt][nt] += a[mt] b[nt], split operands: the small partial products first.  APART: summed from zero and then added, because the
// tensor core's sums are not rounded to nearest (RWKV-5 fp32 B2 T333: error of y 5.9e-7 -> 1.6e-7
// of the norm, 4.4e-7 token by token; bf16 results show no difference)
template <bool APART, int MT, int NA, int NB>
__device__ __forceinline__ void mma_split(float (&c)[MT][2][4], const uint32_t (&a)[MT][NA][4], const uint32_t (&b)[NB][4]) {
    float x[MT][2][4];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            x[mt][0][e] = APART ? 0.f : c[mt][0][e];
            x[mt][1][e] = APART ? 0.f : c[mt][1][e];
        }
#pragma unroll
    for (int order = (NA > 1 ? 2 : 0) + (NB > 1 ? 2 : 0); order >= 0; --order) {
        if (order > 2) continue;
#pragma unroll
        for (int pa = 0; pa < NA; ++pa) {
            const int pb = order - pa;
            if (pb < 0 || pb >= NB) continue;
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                mma(x[mt][0], a[mt][pa], b[pb][0], b[pb][1]);
                mma(x[mt][1], a[mt][pa], b[pb][2], b[pb][3]);
            }
        }
    }
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            c[mt][0][e] = APART ? c[mt][0][e] + x[mt][0][e] : x[mt][0][e];
            c[mt][1][e] = APART ? c[mt][1][e] + x[mt][1][e] : x[mt][1][e];
        }
}
// x = sum of three bf16 numbers, two values at a time (the first in the low half)
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}
__device__ __forceinline__ float bf16_lo(uint32_t x) { return __uint_as_float(x << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t x) { return __uint_as_float(x & 0xffff0000u); }
// x - h with h as a bf16 operand of the multiply-add (exact; 14.7 clocks per split3 and scheduler, 19.1 with h unpacked first)
__device__ __forceinline__ void less_bf16(float& x0, float& x1, uint32_t h) {
    asm("{.reg .b16 a, b, c; mov.b32 {a, b}, %2; mov.b16 c, 0xBF80; fma.rn.f32.bf16 %0, a, c, %0; fma.rn.f32.bf16 %1, b, c, %1;}" : "+f"(x0), "+f"(x1) : "r"(h));
}
__device__ __forceinline__ void split3(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
    h = pack_bf16(x0, x1);
    less_bf16(x0, x1, h);
    m = pack_bf16(x0, x1);
    less_bf16(x0, x1, m);
    l = pack_bf16(x0, x1);
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ void prefetch_l2(const void* p) {   // the line that holds *p
    asm volatile("prefetch.global.L2 [%0];" ::"l"(__cvta_generic_to_global(p) & ~(size_t)127));
}

// ---- two neighbouring channels of a token, as loaded and decoded --------------------------------------------------------------
template <typename E> struct PairOf;
template <> struct PairOf<bf16> { using T = uint32_t; };
template <> struct PairOf<float> { using T = float2; };
template <typename E> using Pair = typename PairOf<E>::T;
__device__ __forceinline__ uint32_t read_pair(const bf16* p, bool vec) {
    if (vec) return __ldg(reinterpret_cast<const uint32_t*>(p));
    const unsigned short* q = reinterpret_cast<const unsigned short*>(p);
    return (uint32_t)__ldg(q) | (uint32_t)__ldg(q + 1) << 16;
}
__device__ __forceinline__ float2 read_pair(const float* p, bool vec) {
    return vec ? __ldg(reinterpret_cast<const float2*>(p)) : make_float2(__ldg(p), __ldg(p + 1));
}
__device__ __forceinline__ float2 decode(uint32_t x) { return make_float2(bf16_lo(x), bf16_hi(x)); }
__device__ __forceinline__ float2 decode(float2 x) { return x; }
template <typename E> __device__ __forceinline__ Pair<E> no_pair();
template <> __device__ __forceinline__ uint32_t no_pair<bf16>() { return 0u; }
template <> __device__ __forceinline__ float2 no_pair<float>() { return make_float2(0.f, 0.f); }
template <typename E> __device__ __forceinline__ bool vec_ok(const E* p, int elements) { return (reinterpret_cast<uintptr_t>(p) & (elements * sizeof(E) - 1)) == 0; }
// rows t0 .. t0 + R - 1 of two channels (one test of the alignment for all of them)
template <typename E, int R>
__device__ __forceinline__ void read_rows(Pair<E> (&x)[R], const E* p, int t0, int n, int C, bool vec) {
    p += (i64)t0 * C;
    if (vec) {
#pragma unroll
        for (int i = 0; i < R; ++i) x[i] = t0 + i < n ? read_pair(p + i * C, true) : no_pair<E>();
    } else {
#pragma unroll
        for (int i = 0; i < R; ++i) x[i] = t0 + i < n ? read_pair(p + i * C, false) : no_pair<E>();
    }
}
// rows g, g + 8, g + 16, g + 24 of four channels
__device__ __forceinline__ void read_four(uint32_t& lo, uint32_t& hi, const bf16* p) {
    const uint2 x = __ldg(reinterpret_cast<const uint2*>(p));
    lo = x.x; hi = x.y;
}
__device__ __forceinline__ void read_four(float2& lo, float2& hi, const float* p) {
    const float4 x = __ldg(reinterpret_cast<const float4*>(p));
    lo = make_float2(x.x, x.y); hi = make_float2(x.z, x.w);
}
template <typename E>
__device__ __forceinline__ void read_eights(Pair<E> (&x)[2][4], const E* p, int g, int n, int C, bool vec) {
    p += (i64)g * C;
#pragma unroll
    for (int b = 0; b < 4; ++b) x[0][b] = x[1][b] = no_pair<E>();
    if (vec) {
#pragma unroll
        for (int b = 0; b < 4; ++b)
            if (g + 8 * b < n) read_four(x[0][b], x[1][b], p + 8 * b * C);
    } else {
#pragma unroll
        for (int b = 0; b < 4; ++b)
            if (g + 8 * b < n) { x[0][b] = read_pair(p + 8 * b * C, false); x[1][b] = read_pair(p + 8 * b * C + 2, false); }
    }
}

__device__ __forceinline__ uint32_t pair_at(int row, int pair) { return img_at(row, 2 * (pair >> 3) + (pair & 1)) + ((pair >> 1) & 3) * 4; }
// eight channels as loaded
__device__ __forceinline__ void put_eight(unsigned char* img, int row, int eight, uint4 x) {
    *reinterpret_cast<uint2*>(img + img_at(row, eight & ~1) + 8 * (eight & 1)) = make_uint2(x.x, x.z);
    *reinterpret_cast<uint2*>(img + img_at(row, eight | 1) + 8 * (eight & 1)) = make_uint2(x.y, x.w);
}
// images of a tensor as it came: bf16 one image, fp32 three
template <typename E> constexpr int kParts = sizeof(E) == 2 ? 1 : 3;
template <typename E>
__device__ __forceinline__ void put_pair(unsigned char* img, int row, int lane, Pair<E> x);   // channels 2 lane, 2 lane + 1
template <>
__device__ __forceinline__ void put_pair<bf16>(unsigned char* img, int row, int lane, uint32_t x) {
    *reinterpret_cast<uint32_t*>(img + pair_at(row, lane)) = x;
}
__device__ __forceinline__ void put_split(unsigned char* img, int row, int lane, float x, float y) {
    uint32_t h, m, l;
    split3(x, y, h, m, l);
    unsigned char* p = img + pair_at(row, lane);
    *reinterpret_cast<uint32_t*>(p) = h;
    *reinterpret_cast<uint32_t*>(p + kImg) = m;
    *reinterpret_cast<uint32_t*>(p + 2 * kImg) = l;
}
template <>
__device__ __forceinline__ void put_pair<float>(unsigned char* img, int row, int lane, float2 x) { put_split(img, row, lane, x.x, x.y); }

// sums that are 0 unless one of the values is not finite
__device__ __forceinline__ void check(float& bad, float2 x) { bad = fmaf(x.y, 0.f, fmaf(x.x, 0.f, bad)); }

// are the logarithms of two decays beyond a limit, or no numbers?
__device__ __forceinline__ bool beyond(float2 l, float limit) { return !(l.x >= -limit && l.y >= -limit); }

// log2 of the decays of two channels, from their raw inputs
__device__ __forceinline__ float2 log2_decay(float2 w) { return make_float2(-kLog2e * ex2(kLog2e * w.x), -kLog2e * ex2(kLog2e * w.y)); }
__device__ __forceinline__ float2 log2_decay_static(float2 w) { return make_float2(-kLog2e * expf(w.x), -kLog2e * expf(w.y)); }

// fp32: a static decay to a power, exp(-e)^m, m of either sign.  The rounding of e m is put back, which the exponential would make large
// (error of y at decays of 0.55 to 0.65 per token 1.5e-7 of its norm, 1.1e-7 with it, token by token 9e-8; inputs w of -6 to -1: 1.9e-7 -> 1.8e-7, 5.2e-7)
__device__ __forceinline__ float decay_power(float e, int m) {
    const float x = (float)m, p = e * x, f = expf(-p);
    return fmaf(f, -fmaf(e, x, -p), f);
}
__device__ __forceinline__ float reciprocal(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// From `rows` (make_operands): what a token's r is scaled by, and k of the token before it
template <bool POWERS> __device__ __forceinline__ float scale_r(float x) { return POWERS ? x : ex2(x); }
template <bool POWERS> __device__ __forceinline__ float scale_k(float x) { return POWERS ? reciprocal(x) : ex2(-x); }

// ---- operands of a segment ---------------------------------------------------------------------------------------------------
// 128 threads: channels 2 lane, 2 lane + 1 of the tokens 8 warp ..  Leaves the images of r~, k~, the bonus sums, S's and D's factors
// and (ROWS) exp(L_{t-1} - L_m) as rows (POWERS; else its log2), row 32: the end.  False (for all
// threads): decays out of range, nothing left.  odd: this thread has seen something else that leaves the segment to the other kernels.
struct Operands {
    unsigned char R[3 * kImg], K[3 * kImg];
    float tot[4 * kN], ruk[kSeg], em[kN], em2[kN];
};
template <typename E, bool STATIC, bool ROWS>
__device__ __forceinline__ bool make_operands(Operands& o, float* rows, int tid, int n, int C, const E* __restrict__ r_, const E* __restrict__ k_,
                                              const E* __restrict__ w_, const E* __restrict__ u_, bool& odd) {
    const int lane = tid & 31, q = tid >> 5, c = 2 * lane, t0 = 8 * q;
    Pair<E> rr[8], kk[8], ww[STATIC ? 1 : 8];
    const bool vec = vec_ok(r_, 2) && vec_ok(k_, 2) && vec_ok(w_, 2);
    read_rows<E, 8>(rr, r_ + c, t0, n, C, vec);
    read_rows<E, 8>(kk, k_ + c, t0, n, C, vec);
    if constexpr (!STATIC) read_rows<E, 8>(ww, w_ + c, t0, n, C, vec);
    else ww[0] = read_pair(w_ + c, vec);
    const float2 u = decode(read_pair(u_ + c, vec_ok(u_, 2)));
    constexpr bool POWERS = STATIC && sizeof(E) == 4;
    const int mid = min(n, kSeg / 2);
    float2 d[STATIC ? 1 : 8], pre, rate, lm, le;   // log2 decays; L before the first of these tokens, L at the middle, L from there to the end
    if constexpr (STATIC) {
        d[0] = log2_decay_static(decode(ww[0]));
        const float nm = (float)mid, ne = (float)(n - mid);
        lm = make_float2(d[0].x * nm, d[0].y * nm);
        le = make_float2(d[0].x * ne, d[0].y * ne);
        const float2 w = decode(ww[0]);
        rate = make_float2(expf(w.x), expf(w.y));
        if (POWERS) pre = make_float2(decay_power(rate.x, min(t0, n) - mid), decay_power(rate.y, min(t0, n) - mid));
    } else {
        float2 s = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            d[i] = t0 + i < n ? log2_decay(decode(ww[i])) : make_float2(0.f, 0.f);
            s.x += d[i].x; s.y += d[i].y;
        }
        *reinterpret_cast<float2*>(o.tot + q * kN + c) = s;
        if (__syncthreads_or(beyond(s, kRange))) return false;   // (eight tokens alone are too much)
        float2 t[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) t[i] = *reinterpret_cast<const float2*>(o.tot + i * kN + c);
        lm = make_float2(t[0].x + t[1].x, t[0].y + t[1].y);
        le = make_float2(t[2].x + t[3].x, t[2].y + t[3].y);
        pre = q == 0 ? make_float2(-lm.x, -lm.y) : q == 1 ? make_float2(-t[1].x, -t[1].y) : q == 2 ? make_float2(0.f, 0.f) : t[2];
    }
    float bad = 0.f, x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float2 a, b;   // L before and after the token, from the middle; the decay there (POWERS)
        if constexpr (POWERS) {
            const int behind = min(t0 + i + 1, n) - mid;
            a = pre;
            b = pre = make_float2(decay_power(rate.x, behind), decay_power(rate.y, behind));
        } else if constexpr (STATIC) {
            const float ta = (float)(min(t0 + i, n) - mid), tb = (float)(min(t0 + i + 1, n) - mid);
            a = make_float2(d[0].x * ta, d[0].y * ta);
            b = make_float2(d[0].x * tb, d[0].y * tb);
        } else {
            a = pre;
            b = pre = make_float2(pre.x + d[i].x, pre.y + d[i].y);
        }
        if (ROWS) *reinterpret_cast<float2*>(rows + (t0 + i) * kRld + c) = a;
        const float2 r = decode(rr[i]), k = decode(kk[i]);
        const float2 rs = make_float2(r.x * scale_r<POWERS>(a.x), r.y * scale_r<POWERS>(a.y)), ks = make_float2(k.x * scale_k<POWERS>(b.x), k.y * scale_k<POWERS>(b.y));
        check(bad, rs); check(bad, ks);
        put_split(o.R, t0 + i, lane, rs.x, rs.y);
        put_split(o.K, t0 + i, lane, ks.x, ks.y);
        x[i] = fmaf(r.x * u.x, k.x, r.y * u.y * k.y);
        if (ROWS && q == 3 && i == 7) *reinterpret_cast<float2*>(rows + kSeg * kRld + c) = b;
    }
    float s = reduce8(x, lane);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if ((lane & 3) == 0) o.ruk[t0 + (lane >> 2)] = s;
    if (q == 0) {
        if constexpr (POWERS) {
            *reinterpret_cast<float2*>(o.em + c) = make_float2(decay_power(rate.x, mid), decay_power(rate.y, mid));
            *reinterpret_cast<float2*>(o.em2 + c) = make_float2(decay_power(rate.x, n - mid), decay_power(rate.y, n - mid));
        } else {
            *reinterpret_cast<float2*>(o.em + c) = make_float2(ex2(lm.x), ex2(lm.y));
            *reinterpret_cast<float2*>(o.em2 + c) = make_float2(ex2(le.x), ex2(le.y));
        }
    }
    check(bad, make_float2(s, 0.f));
    odd = bad != 0.f || (!STATIC && (beyond(lm, kRange) || beyond(le, kRange)));
    return true;
}
// the images of a tensor as it came (pieces of 16 bytes where the alignment allows)
template <typename E>
__device__ __forceinline__ bool stage_images(unsigned char* img, int tid, int n, int C, const E* __restrict__ x_) {
    float bad = 0.f;
    const int lane = tid & 31, t0 = 8 * (tid >> 5);
    if (sizeof(E) == 2 && vec_ok(x_, 8)) {
        uint4 x[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int row = 16 * i + (tid >> 3);
            x[i] = row < n ? __ldg(reinterpret_cast<const uint4*>(x_ + (i64)row * C + 8 * (tid & 7))) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            put_eight(img, 16 * i + (tid >> 3), tid & 7, x[i]);
            check(bad, decode(x[i].x)); check(bad, decode(x[i].y)); check(bad, decode(x[i].z)); check(bad, decode(x[i].w));
        }
    } else {
        Pair<E> x[8];
        read_rows<E, 8>(x, x_ + 2 * lane, t0, n, C, vec_ok(x_, 2));
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            check(bad, decode(x[i]));
            put_pair<E>(img, t0 + i, lane, x[i]);
        }
    }
    return bad != 0.f;
}

// Token x token products: c = rows 16 mt .. of one set of images times rows 16 nt .. of another, over the 64 channels (two sums side
// by side: the products of one sum wait for one another)
template <bool APART, int NA, int NB>
__device__ __forceinline__ void gram(float (&c)[1][2][4], const unsigned char* a_img, const unsigned char* b_img, int mt, int nt, int lane) {
    float c2[1][2][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) c[0][0][e] = c[0][1][e] = c2[0][0][e] = c2[0][1][e] = 0.f;
#pragma unroll
    for (int kk = 0; kk < 4; kk += 2) {
        uint32_t a[1][NA][4], b[NB][4], a2[1][NA][4], b2[NB][4];
        ldsm<NA>(a[0], smem_addr(a_img) + frag_rows(16 * mt, 2 * kk, lane));
        ldsm<NB>(b, smem_addr(b_img) + frag_cols(16 * nt, 2 * kk, lane));
        ldsm<NA>(a2[0], smem_addr(a_img) + frag_rows(16 * mt, 2 * kk + 2, lane));
        ldsm<NB>(b2, smem_addr(b_img) + frag_cols(16 * nt, 2 * kk + 2, lane));
        mma_split<APART, 1, NA, NB>(c, a, b);
        mma_split<APART, 1, NA, NB>(c2, a2, b2);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) { c[0][0][e] += c2[0][0][e]; c[0][1][e] += c2[0][1][e]; }
}

// Triangular token x token matrices: three images of the tiles (0,0), (0,1) or (1,0), (1,1) at mt + nt, rows of two 16-byte pieces
__device__ __forceinline__ uint32_t tile_at(int tile, int row, int piece) { return tile * 512 + row * 32 + ((piece ^ ((row >> 2) & 1)) << 4); }
// a pair of row `row`, columns 8 j + 2 q, + 1 of a tile
__device__ __forceinline__ void put_tile(unsigned char* img, int tile, int row, int j, int q, float x, float y) {
    uint32_t h, m, l;
    split3(x, y, h, m, l);
    unsigned char* p = img + tile_at(tile, row, j) + 4 * q;
    *reinterpret_cast<uint32_t*>(p) = h;
    *reinterpret_cast<uint32_t*>(p + kTiles) = m;
    *reinterpret_cast<uint32_t*>(p + 2 * kTiles) = l;
}
// Fragments of a transposed tile (rows t0 + .., columns s0 + ..), each element times t - 1 - s
__device__ __forceinline__ void weigh_by_distance(uint32_t (&w)[3][4], const uint32_t (&f)[3][4], int t0, int s0, int lane) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float d = (float)(t0 + (lane >> 2) + 8 * (i & 1) - 1 - (s0 + 2 * (lane & 3) + 8 * (i >> 1)));
        const float x = bf16_lo(f[0][i]) + (bf16_lo(f[1][i]) + bf16_lo(f[2][i])), z = bf16_hi(f[0][i]) + (bf16_hi(f[1][i]) + bf16_hi(f[2][i]));
        split3(x * d, z * (d - 1.f), w[0][i], w[1][i], w[2][i]);
    }
}
template <bool TRANS>   // a tile as A fragments, as stored or transposed
__device__ __forceinline__ void tile_frag(uint32_t (&f)[3][4], const unsigned char* img, int tile, int lane) {
    if (TRANS) ldsm_t<3, kTiles>(f, smem_addr(img) + tile_at(tile, (lane & 7) + ((lane >> 4) << 3), (lane >> 3) & 1));
    else ldsm<3, kTiles>(f, smem_addr(img) + tile_at(tile, lane & 15, lane >> 4));
}

// four neighbouring channels out of two accumulator tiles
__device__ __forceinline__ void store_four(bf16* p, float x0, float x1, float x2, float x3, bool vec) {
    const uint2 v = make_uint2(pack_bf16(x0, x1), pack_bf16(x2, x3));
    if (vec) *reinterpret_cast<uint2*>(p) = v;
    else {
        unsigned short* s = reinterpret_cast<unsigned short*>(p);
        s[0] = (unsigned short)v.x; s[1] = (unsigned short)(v.x >> 16); s[2] = (unsigned short)v.y; s[3] = (unsigned short)(v.y >> 16);
    }
}
__device__ __forceinline__ void store_four(float* p, float x0, float x1, float x2, float x3, bool vec) {
    if (vec) *reinterpret_cast<float4*>(p) = make_float4(x0, x1, x2, x3);
    else { p[0] = x0; p[1] = x1; p[2] = x2; p[3] = x3; }
}

// Asks L2 for what the block `ahead` places further on will read first: rows of up to five tensors, a state or two (128 lines each)
template <typename E>
__device__ __forceinline__ void prefetch_rows(const E* x, i64 base, int n, int C, int row) {
    if (row < n) {
        prefetch_l2(x + base + (i64)row * C);
        if (sizeof(E) == 4) prefetch_l2(x + base + (i64)row * C + 32);
    }
}

// A read that stays where it is written: the states are asked for a step before they are used, which the compiler would undo
__device__ __forceinline__ float4 read_now(const float* p) {
    float4 x;
    asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "l"(p));
    return x;
}

// ---- kernels -----------------------------------------------------------------------------------------------------------------
// y of a segment from its start state.  One block per (unit, segment), 4 warps; a warp has 16 values of all tokens.
template <typename E>
struct YSmem {
    Operands o;
    unsigned char V[kParts<E> * kImg];
    unsigned char M[3 * kTiles];   // A transposed: [t][s]
};
template <typename E, bool STATIC>
__global__ void __launch_bounds__(128, 5) seg_mma_y_kernel(int T, int H, int nseg, const E* __restrict__ r_, const E* __restrict__ k_,
                                                           const E* __restrict__ v_, const E* __restrict__ w_, const E* __restrict__ u_,
                                                           const float* __restrict__ states, E* __restrict__ y_, int* __restrict__ flags, bool known, int ahead) {
    extern __shared__ __align__(128) unsigned char smem_seg_y[];
    YSmem<E>& sm = *reinterpret_cast<YSmem<E>*>(smem_seg_y);
    constexpr int NV = kParts<E>;
    const i64 unit = blockIdx.x / nseg;
    const int seg = blockIdx.x % nseg, h = unit % H, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, C = H * kN;
    const int g = lane >> 2, q = lane & 3, n = min(kSeg, T - seg * kSeg);
    const i64 base = (unit / H * T + (i64)seg * kSeg) * C + h * kN;
    if (known && flags[blockIdx.x]) return;
    if (blockIdx.x + ahead < gridDim.x) {
        const i64 next = blockIdx.x + ahead;
        const int seg1 = next % nseg, h1 = next / nseg % H, n1 = min(kSeg, T - seg1 * kSeg);
        const i64 base1 = (next / nseg / H * T + (i64)seg1 * kSeg) * C + h1 * kN;
        const E* x = warp == 0 ? r_ : warp == 1 ? k_ : warp == 2 ? v_ : w_;
        if (!STATIC || warp < 3) prefetch_rows(x, base1, n1, C, lane);
        prefetch_l2(states + next * kN * kN + tid * 32);
    }
    float S[4][2][4];   // [16 keys][8 values] as B fragments
    {
        const float* p = states + (i64)blockIdx.x * kN * kN + 16 * warp + at16(g);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[kk][nt][e] = p[(16 * kk + 4 * q + e) * kN + 2 * nt];
    }
    bool bad;
    if (!make_operands<E, STATIC, false>(sm.o, nullptr, tid, n, C, r_ + base, k_ + base, w_ + (STATIC ? h * kN : base), u_ + h * kN, bad)) {
        if (tid == 0) flags[blockIdx.x] = 1;
        return;
    }
    bad |= stage_images<E>(sm.V, tid, n, C, v_ + base);
    if (__syncthreads_or(bad)) {
        if (tid == 0) flags[blockIdx.x] = 1;
        return;
    }
    // A: three of the warps a 16 x 16 tile each, and which three turns with the block (a warp's number is its scheduler)
    const int job = (warp + blockIdx.x) & 3;
    if (job < 3) {
        const int mt = job > 0, nt = job > 1;
        float c[1][2][4];
        gram<sizeof(E) == 4, 3, 3>(c, sm.o.R, sm.o.K, mt, nt, lane);
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int t = 16 * mt + g + 8 * e, s = 16 * nt + 8 * j + 2 * q;
                const float x = s < t ? c[0][j][2 * e] : s == t ? sm.o.ruk[t] : 0.f, z = s + 1 < t ? c[0][j][2 * e + 1] : s + 1 == t ? sm.o.ruk[t] : 0.f;
                put_tile(sm.M, mt + nt, g + 8 * e, j, q, x, z);
            }
    }
    float acc[2][2][4];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[mt][0][e] = acc[mt][1][e] = 0.f;
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
        uint32_t a[2][3][4], b[3][4];
        const float4 f = *reinterpret_cast<const float4*>(sm.o.em + 16 * kk + 4 * q);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            split3(S[kk][nt][0] * f.x, S[kk][nt][1] * f.y, b[0][2 * nt], b[1][2 * nt], b[2][2 * nt]);
            split3(S[kk][nt][2] * f.z, S[kk][nt][3] * f.w, b[0][2 * nt + 1], b[1][2 * nt + 1], b[2][2 * nt + 1]);
        }
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) ldsm<3>(a[mt], smem_addr(sm.o.R) + frag_rows(16 * mt, 2 * kk, lane));
        mma_split<sizeof(E) == 4, 2, 3, 3>(acc, a, b);
    }
    __syncthreads();
#pragma unroll
    for (int kt = 0; kt < 2; ++kt) {
        uint32_t b[NV][4];
        ldsm_t<NV>(b, smem_addr(sm.V) + frag_rows(16 * kt, 2 * warp, lane));
#pragma unroll
        for (int mt = kt; mt < 2; ++mt) {
            uint32_t a[1][3][4];
            tile_frag<false>(a[0], sm.M, mt + kt, lane);
            float(&c)[1][2][4] = *reinterpret_cast<float(*)[1][2][4]>(&acc[mt]);
            mma_split<sizeof(E) == 4, 1, 3, NV>(c, a, b);
        }
    }
    const bool vec = vec_ok(y_, 4);
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int t = 16 * mt + g + 8 * e;
            if (t < n) store_four(y_ + base + (i64)t * C + 16 * warp + 4 * q, acc[mt][0][2 * e], acc[mt][0][2 * e + 1], acc[mt][1][2 * e], acc[mt][1][2 * e + 1], vec);
        }
    float wrong = 0.f;
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int e = 0; e < 4; ++e) check(wrong, make_float2(acc[mt][0][e], acc[mt][1][e]));
    bad = __syncthreads_or(wrong != 0.f);   // a state that is not finite, or a product that left the range of fp32
    if (tid == 0) flags[blockIdx.x] = bad;
}

// Gradients of a segment from its start state S and the adjoint D behind it.  One block per (unit, segment), 4 warps; a warp has
// 16 keys (gr, gk, gw, gu) and 16 values (gv) of all tokens.  STATIC: out2 = partials (gw, gu) of the segment, rows of 2 C.
template <typename E>
struct BwdSmemM {
    Operands o;
    unsigned char V[kParts<E> * kImg], G[kParts<E> * kImg];
    unsigned char A[3 * kTiles], Gm[3 * kTiles];
    float rows[(kSeg + 1) * kRld], gamma[kSeg], a0[kN];
};
template <typename E, bool STATIC>
__global__ void __launch_bounds__(128, sizeof(E) == 2 ? 4 : 3)
    seg_mma_backward_kernel(int T, int H, int nseg, const E* __restrict__ r_, const E* __restrict__ k_, const E* __restrict__ v_,
                            const E* __restrict__ w_, const E* __restrict__ u_, const E* __restrict__ gy_, const float* __restrict__ S_,
                            const float* __restrict__ D_, E* __restrict__ gr_, E* __restrict__ gk_, E* __restrict__ gv_, E* __restrict__ gw_,
                            float* __restrict__ partial_, const int* __restrict__ left, int* __restrict__ flags, int ahead) {
    extern __shared__ __align__(128) unsigned char smem_seg_b[];
    BwdSmemM<E>& sm = *reinterpret_cast<BwdSmemM<E>*>(smem_seg_b);
    constexpr int NV = kParts<E>;
    constexpr bool WEIGHTS = STATIC && sizeof(E) == 4, POWERS = WEIGHTS;   // see dL/dlog d above (bf16: its rounding is a thousand times what cancels)
    const i64 unit = blockIdx.x / nseg;
    const int seg = blockIdx.x % nseg, h = unit % H, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, C = H * kN;
    const int g = lane >> 2, q = lane & 3, n = min(kSeg, T - seg * kSeg);
    const i64 base = (unit / H * T + (i64)seg * kSeg) * C + h * kN;
    if (left != nullptr && left[blockIdx.x]) {
        if (tid == 0) flags[blockIdx.x] = 1;
        return;
    }
    if (blockIdx.x + ahead < gridDim.x) {
        const i64 next = blockIdx.x + ahead;
        const int seg1 = next % nseg, h1 = next / nseg % H, n1 = min(kSeg, T - seg1 * kSeg);
        const i64 base1 = (next / nseg / H * T + (i64)seg1 * kSeg) * C + h1 * kN;
        const E* x = warp == 0 ? r_ : warp == 1 ? k_ : warp == 2 ? v_ : gy_;
        prefetch_rows(x, base1, n1, C, lane);
        if (!STATIC && warp == 0) prefetch_rows(w_, base1, n1, C, lane);
        prefetch_l2(S_ + next * kN * kN + tid * 32);
        prefetch_l2(D_ + next * kN * kN + tid * 32);
    }
    float D[4][2][4];   // [16 keys][8 values] as B fragments
    {
        const float* p = D_ + (i64)blockIdx.x * kN * kN + 16 * warp + at16(g);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) D[kk][nt][e] = p[(16 * kk + 4 * q + e) * kN + 2 * nt];
    }
    bool bad;
    if (!make_operands<E, STATIC, true>(sm.o, sm.rows, tid, n, C, r_ + base, k_ + base, w_ + (STATIC ? h * kN : base), u_ + h * kN, bad)) {
        if (tid == 0) flags[blockIdx.x] = 1;
        return;
    }
    bad |= stage_images<E>(sm.V, tid, n, C, v_ + base);
    bad |= stage_images<E>(sm.G, tid, n, C, gy_ + base);
    if (__syncthreads_or(bad)) {
        if (tid == 0) flags[blockIdx.x] = 1;
        return;
    }
    const bool vec = vec_ok(gr_, 4) && vec_ok(gk_, 4) && vec_ok(gv_, 4) && (STATIC || vec_ok(gw_, 4));
    // the two token x token matrices, 16 x 16 tiles (0,0), (0,1), (1,1): A six partial products each; G one (bf16) or six (fp32)
    for (int job = (warp + blockIdx.x) & 3; job < 6; job = job >= 3 && NV == 1 ? job + 1 : NV == 1 ? 6 : job + 4) {
        const int tile = job % 3, mt = tile > 1, nt = tile > 0;
        float c[1][2][4];
        if (job < 3) gram<sizeof(E) == 4, 3, 3>(c, sm.o.K, sm.o.R, mt, nt, lane);
        else gram<sizeof(E) == 4, NV, NV>(c, sm.V, sm.G, mt, nt, lane);
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int s = 16 * mt + g + 8 * e, t = 16 * nt + 8 * j + 2 * q;
                const float x = c[0][j][2 * e], z = c[0][j][2 * e + 1];
                const bool diag = job < 3;
                if (!diag && s == t) sm.gamma[s] = x;
                if (!diag && s == t + 1) sm.gamma[s] = z;
                put_tile(diag ? sm.A : sm.Gm, mt + nt, g + 8 * e, j, q, s < t ? x : diag && s == t ? sm.o.ruk[s] : 0.f,
                         s < t + 1 ? z : diag && s == t + 1 ? sm.o.ruk[s] : 0.f);
            }
    }
    float wrong = 0.f;
    const i64 so = (i64)blockIdx.x * kN * kN + (16 * warp + at16(g)) * kN + 4 * q;
    float4 s4[2][2], x4[2][2];   // S and D of 16 values: of this step and of the next, [tile]
    auto read_states = [&](int kk) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            s4[kk & 1][nt] = read_now(S_ + so + 2 * nt * kN + 16 * kk);
            x4[kk & 1][nt] = read_now(D_ + so + 2 * nt * kN + 16 * kk);
        }
    };
    {   // gv = K~ D' + A gY
        float acc[2][2][4];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[mt][0][e] = acc[mt][1][e] = 0.f;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            uint32_t a[2][3][4], b[3][4];
            const float4 f = *reinterpret_cast<const float4*>(sm.o.em2 + 16 * kk + 4 * q);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                split3(D[kk][nt][0] * f.x, D[kk][nt][1] * f.y, b[0][2 * nt], b[1][2 * nt], b[2][2 * nt]);
                split3(D[kk][nt][2] * f.z, D[kk][nt][3] * f.w, b[0][2 * nt + 1], b[1][2 * nt + 1], b[2][2 * nt + 1]);
            }
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) ldsm<3>(a[mt], smem_addr(sm.o.K) + frag_rows(16 * mt, 2 * kk, lane));
            mma_split<sizeof(E) == 4, 2, 3, 3>(acc, a, b);
        }
        read_states(0);
        __syncthreads();
#pragma unroll
        for (int kt = 0; kt < 2; ++kt) {
            uint32_t b[NV][4];
            ldsm_t<NV>(b, smem_addr(sm.G) + frag_rows(16 * kt, 2 * warp, lane));
#pragma unroll
            for (int mt = 0; mt <= kt; ++mt) {
                uint32_t a[1][3][4];
                tile_frag<false>(a[0], sm.A, mt + kt, lane);
                float(&c)[1][2][4] = *reinterpret_cast<float(*)[1][2][4]>(&acc[mt]);
                mma_split<sizeof(E) == 4, 1, 3, NV>(c, a, b);
            }
        }
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int t = 16 * mt + g + 8 * e;
                if (t < n) store_four(gv_ + base + (i64)t * C + 16 * warp + 4 * q, acc[mt][0][2 * e], acc[mt][0][2 * e + 1], acc[mt][1][2 * e], acc[mt][1][2 * e + 1], vec);
                check(wrong, make_float2(acc[mt][0][2 * e], acc[mt][0][2 * e + 1]));
                check(wrong, make_float2(acc[mt][1][2 * e], acc[mt][1][2 * e + 1]));
            }
    }
    // dk~ = V D'^T + G R~, dr~ = gY S'^T + G^T K~
    const int c = 16 * warp + 4 * q;   // this lane's four keys: two of each tile
    Pair<E> rp[2][4], kp[2][4];        // [two keys][eight tokens]
    float dk[2][2][4], dr[2][2][4], a0[2] = {0.f, 0.f};
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) dk[mt][nt][e] = dr[mt][nt][e] = 0.f;
    {
        float fs[2], fd[2];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) { fs[nt] = sm.o.em[16 * warp + at16(g) + 2 * nt]; fd[nt] = sm.o.em2[16 * warp + at16(g) + 2 * nt]; }
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            uint32_t bs[3][4], bd[3][4];
            if (kk < 3) read_states(kk + 1);
            else {
                read_eights<E>(rp, r_ + base + c, g, n, C, vec_ok(r_, 4));
                read_eights<E>(kp, k_ + base + c, g, n, C, vec_ok(k_, 4));
            }
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                float4 s = s4[kk & 1][nt], x = x4[kk & 1][nt];
                s.x *= fs[nt]; s.y *= fs[nt]; s.z *= fs[nt]; s.w *= fs[nt];
                x.x *= fd[nt]; x.y *= fd[nt]; x.z *= fd[nt]; x.w *= fd[nt];
                a0[nt] = fmaf(s.x, x.x, fmaf(s.y, x.y, fmaf(s.z, x.z, fmaf(s.w, x.w, a0[nt]))));
                split3(s.x, s.y, bs[0][2 * nt], bs[1][2 * nt], bs[2][2 * nt]);
                split3(s.z, s.w, bs[0][2 * nt + 1], bs[1][2 * nt + 1], bs[2][2 * nt + 1]);
                split3(x.x, x.y, bd[0][2 * nt], bd[1][2 * nt], bd[2][2 * nt]);
                split3(x.z, x.w, bd[0][2 * nt + 1], bd[1][2 * nt + 1], bd[2][2 * nt + 1]);
            }
            uint32_t a[2][NV][4];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) ldsm<NV>(a[mt], smem_addr(sm.V) + frag_rows(16 * mt, 2 * kk, lane));
            mma_split<sizeof(E) == 4, 2, NV, 3>(dk, a, bd);
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) ldsm<NV>(a[mt], smem_addr(sm.G) + frag_rows(16 * mt, 2 * kk, lane));
            mma_split<sizeof(E) == 4, 2, NV, 3>(dr, a, bs);
        }
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {   // a0: sum over the values of a key, to the lanes that have its column below
        a0[nt] += __shfl_xor_sync(0xffffffffu, a0[nt], 1);
        a0[nt] += __shfl_xor_sync(0xffffffffu, a0[nt], 2);
        if (q == 0) sm.a0[16 * warp + at16(g) + 2 * nt] = a0[nt];
    }
    __syncwarp();
    float aend[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const float4 l = *reinterpret_cast<const float4*>(sm.rows + (8 * b + g + 1) * kRld + c);
        float2 k0 = decode(kp[0][b]), k1 = decode(kp[1][b]);
        if constexpr (WEIGHTS) {   // the distances to the segment's end, and to its start
            const float4 l0 = *reinterpret_cast<const float4*>(sm.rows + (8 * b + g) * kRld + c);
            const float2 r0 = decode(rp[0][b]), r1 = decode(rp[1][b]);
            const float t = (float)(8 * b + g), d = (float)(n - 1) - t;
            k0.x *= d; k0.y *= d; k1.x *= d; k1.y *= d;
            aend[0] = fmaf(t * r0.x * l0.x, dr[b >> 1][0][2 * (b & 1)], aend[0]);
            aend[1] = fmaf(t * r0.y * l0.y, dr[b >> 1][0][2 * (b & 1) + 1], aend[1]);
            aend[2] = fmaf(t * r1.x * l0.z, dr[b >> 1][1][2 * (b & 1)], aend[2]);
            aend[3] = fmaf(t * r1.y * l0.w, dr[b >> 1][1][2 * (b & 1) + 1], aend[3]);
        }
        aend[0] = fmaf(k0.x * scale_k<POWERS>(l.x), dk[b >> 1][0][2 * (b & 1)], aend[0]);
        aend[1] = fmaf(k0.y * scale_k<POWERS>(l.y), dk[b >> 1][0][2 * (b & 1) + 1], aend[1]);
        aend[2] = fmaf(k1.x * scale_k<POWERS>(l.z), dk[b >> 1][1][2 * (b & 1)], aend[2]);
        aend[3] = fmaf(k1.y * scale_k<POWERS>(l.w), dk[b >> 1][1][2 * (b & 1) + 1], aend[3]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int m = 4; m < 32; m <<= 1) aend[i] += __shfl_xor_sync(0xffffffffu, aend[i], m);
        aend[i] = WEIGHTS ? fmaf((float)n, sm.a0[c + i], aend[i]) : aend[i] + sm.a0[c + i];
    }
    float dw[WEIGHTS ? 2 : 1][2][4];   // sum_s (t - 1 - s) G[s,t] k~_s
    if constexpr (WEIGHTS) {
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int e = 0; e < 4; ++e) dw[mt][0][e] = dw[mt][1][e] = 0.f;
    }
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
        float(&ck)[1][2][4] = *reinterpret_cast<float(*)[1][2][4]>(&dk[mt]);
        float(&cr)[1][2][4] = *reinterpret_cast<float(*)[1][2][4]>(&dr[mt]);
#pragma unroll
        for (int kt = 0; kt < 2; ++kt) {
            uint32_t a[1][3][4], b[3][4];
            if (kt >= mt) {
                tile_frag<false>(a[0], sm.Gm, mt + kt, lane);
                ldsm_t<3>(b, smem_addr(sm.o.R) + frag_rows(16 * kt, 2 * warp, lane));
                mma_split<sizeof(E) == 4, 1, 3, 3>(ck, a, b);
            }
            if (kt <= mt) {
                tile_frag<true>(a[0], sm.Gm, mt + kt, lane);
                ldsm_t<3>(b, smem_addr(sm.o.K) + frag_rows(16 * kt, 2 * warp, lane));
                mma_split<sizeof(E) == 4, 1, 3, 3>(cr, a, b);
                if constexpr (WEIGHTS) {
                    uint32_t d[1][3][4];
                    float(&cw)[1][2][4] = *reinterpret_cast<float(*)[1][2][4]>(&dw[mt]);
                    weigh_by_distance(d[0], a[0], 16 * mt, 16 * kt, lane);
                    mma_split<sizeof(E) == 4, 1, 3, 3>(cw, d, b);
                }
            }
        }
    }
    // per token and key: scales and bonus terms, then the decay gradient
    float P[4][4], x[4][4], gu[4] = {0.f, 0.f, 0.f, 0.f}, gw[4] = {0.f, 0.f, 0.f, 0.f}, u[4];   // [eight tokens][key]; x = Q - P
    {
        const bool vu = vec_ok(u_, 2);
        const float2 u0 = decode(read_pair(u_ + h * kN + c, vu)), u1 = decode(read_pair(u_ + h * kN + c + 2, vu));
        u[0] = u0.x; u[1] = u0.y; u[2] = u1.x; u[3] = u1.y;
    }
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const int mt = b >> 1, e = b & 1, t = 8 * b + g;
        const float4 l0 = *reinterpret_cast<const float4*>(sm.rows + t * kRld + c), l1 = *reinterpret_cast<const float4*>(sm.rows + (t + 1) * kRld + c);
        const float before[4] = {l0.x, l0.y, l0.z, l0.w}, behind[4] = {l1.x, l1.y, l1.z, l1.w}, gm = sm.gamma[t];
        const float2 r0 = decode(rp[0][b]), r1 = decode(rp[1][b]), k0 = decode(kp[0][b]), k1 = decode(kp[1][b]);
        const float r[4] = {r0.x, r0.y, r1.x, r1.y}, k[4] = {k0.x, k0.y, k1.x, k1.y};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float &yk = dk[mt][i >> 1][2 * e + (i & 1)], &yr = dr[mt][i >> 1][2 * e + (i & 1)];
            yk *= scale_k<POWERS>(behind[i]);
            if constexpr (WEIGHTS) {
                const float f = scale_r<POWERS>(before[i]);
                gw[i] = fmaf(r[i] * f, dw[mt][i >> 1][2 * e + (i & 1)], gw[i]);
                yr *= f;
                check(wrong, make_float2(yk, yr));
            } else {
                yr *= scale_r<POWERS>(before[i]);
                P[b][i] = r[i] * yr;
                x[b][i] = fmaf(k[i], yk, -P[b][i]);
            }
            gu[i] = fmaf(gm, r[i] * k[i], gu[i]);
            yk = fmaf(u[i] * r[i], gm, yk);   // (in the order of the token-by-token kernels, which cannot overflow where the result does not)
            yr = fmaf(u[i] * k[i], gm, yr);
        }
    }
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int t = 16 * mt + g + 8 * e;
            const i64 o = base + (i64)t * C + c;
            if (t < n) {
                store_four(gk_ + o, dk[mt][0][2 * e], dk[mt][0][2 * e + 1], dk[mt][1][2 * e], dk[mt][1][2 * e + 1], vec);
                store_four(gr_ + o, dr[mt][0][2 * e], dr[mt][0][2 * e + 1], dr[mt][1][2 * e], dr[mt][1][2 * e + 1], vec);
            }
        }
    Pair<E> wp[2][4];
    if constexpr (!STATIC) read_eights<E>(wp, w_ + base + c, g, n, C, vec_ok(w_, 4));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float after = 0.f;
#pragma unroll
        for (int b = 3; b >= 0 && !WEIGHTS; --b) {   // sums over the tokens from here on: over lanes inside eight tokens, then over the eights
            float s = x[b][i];
#pragma unroll
            for (int m = 1; m < 8; m <<= 1) {
                const float o = __shfl_down_sync(0xffffffffu, s, 4 * m);
                if (g + m < 8) s += o;
            }
            // A_end - sum_{tau > t} (Q - P) - Q_t = A_end - sum_{tau >= t} (Q - P) - P_t
            x[b][i] = aend[i] - (after + s) - P[b][i];
            after += __shfl_sync(0xffffffffu, s, q);
            if (STATIC && 8 * b + g < n) gw[i] += x[b][i];
        }
#pragma unroll
        for (int m = 4; m < 32; m <<= 1) {
            gu[i] += __shfl_xor_sync(0xffffffffu, gu[i], m);
            if (STATIC) gw[i] += __shfl_xor_sync(0xffffffffu, gw[i], m);
        }
        if (WEIGHTS) gw[i] += aend[i];
        // (per-token decays: the sum over all tokens in the first one's; every P and Q of the key is in it, and so every gr and gk)
        check(wrong, make_float2(STATIC ? gw[i] : x[0][i], gu[i]));
    }
    if (g == 0) {
        float* p = partial_ + (unit / H * nseg + seg) * (STATIC ? 2 : 1) * C + h * kN + c;
        if (STATIC) {
#pragma unroll
            for (int i = 0; i < 4; ++i) p[i] = -expf(to_f(w_[h * kN + c + i])) * gw[i];   // d log d / d w_raw = log d
            p += C;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) p[i] = gu[i];
    }
    if constexpr (!STATIC) {
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const float2 w0 = decode(wp[0][b]), w1 = decode(wp[1][b]);
            if (8 * b + g < n)
                store_four(gw_ + base + (i64)(8 * b + g) * C + c, -ex2(kLog2e * w0.x) * x[b][0], -ex2(kLog2e * w0.y) * x[b][1], -ex2(kLog2e * w1.x) * x[b][2],
                           -ex2(kLog2e * w1.y) * x[b][3], vec);
        }
    }
    bad = __syncthreads_or(wrong != 0.f);
    if (tid == 0) flags[blockIdx.x] = bad;
}

// States at the start of every segment (REV: adjoints at the end), one block per unit walking its segments: S <- S diag(f) + k'^T V
// with k'_s = k_s exp(L_end - L_s) (REV: r'_t = r_t exp(L_{t-1}), gy): all factors are at most 1.  Warps 0 to 3 have the state in
// registers, 16 keys each, warps 4 to 11 make the operands of the segments to come (B8 T1000 H32 bf16: 80 us with four of them, two
// sums of products at a time and states stored in pieces of 8 bytes, 65 us now: 3.5 TB/s; a third buffer of
// operands changed nothing).
template <typename E>
struct ChainSmem {
    unsigned char A[3 * kImg], B[kParts<E> * kImg];
    float f[kN], tot[8 * kN];
};
template <int ID>
__device__ __forceinline__ void bar_join(int odd) {
    if (odd) asm volatile("bar.sync %0, 384;" ::"n"(ID + 1) : "memory");
    else asm volatile("bar.sync %0, 384;" ::"n"(ID) : "memory");
}
template <int ID>
__device__ __forceinline__ void bar_tell(int odd) {
    if (odd) asm volatile("bar.arrive %0, 384;" ::"n"(ID + 1) : "memory");
    else asm volatile("bar.arrive %0, 384;" ::"n"(ID) : "memory");
}
// The same walk once more, where a state has come out not finite: as the local sums and the scan do it, in fp32 with one multiply-add
// per token.  (By products the parts of an infinity, and an infinity against a part that is 0, make NaN where these have an infinity.)
template <typename E, bool STATIC, bool REV>
__device__ __noinline__ void walk_again(int T, int nseg, int C, const E* a_, const E* b_, const E* w_, float* states) {
    const int j = threadIdx.x >> 2, i0 = 16 * (threadIdx.x & 3);   // a key, 16 values
    if (j >= kN) return;
    float S[16], c[16], lw = 0.f, f;
#pragma unroll
    for (int i = 0; i < 16; ++i) S[i] = 0.f;
    if (STATIC) lw = -expf(to_f(w_[j]));
    for (int it = 0; it < nseg; ++it) {
        const int seg = REV ? nseg - 1 - it : it, n = min(kSeg, T - seg * kSeg);
        float* p = states + (i64)seg * kN * kN + j * kN + i0;
        f = 1.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) { p[i] = S[i]; c[i] = 0.f; }
        for (int q = 0; q < n; ++q) {
            const i64 o = ((i64)seg * kSeg + (REV ? q : n - 1 - q)) * C;
            if (STATIC) f = q == 0 ? 1.f : expf(lw * (float)q);
            const float a = to_f(a_[o + j]) * f;
#pragma unroll
            for (int i = 0; i < 16; ++i) c[i] = fmaf(a, to_f(b_[o + i0 + i]), c[i]);
            if (!STATIC) f *= expf(-expf(to_f(w_[o + j])));
        }
        if (STATIC) f = expf(lw * (float)n);
#pragma unroll
        for (int i = 0; i < 16; ++i) S[i] = fmaf(S[i], f, c[i]);
    }
}
template <typename E, bool STATIC, bool REV>
__global__ void __launch_bounds__(384, sizeof(E) == 2 ? 2 : 1) seg_mma_chain_kernel(int T, int H, int nseg, const E* __restrict__ a_, const E* __restrict__ b_,
                                                               const E* __restrict__ w_, float* __restrict__ states, int* __restrict__ flags) {
    extern __shared__ __align__(128) unsigned char smem_seg_c[];
    ChainSmem<E>* buf = reinterpret_cast<ChainSmem<E>*>(smem_seg_c);
    constexpr int NV = kParts<E>;
    const i64 unit = blockIdx.x;
    const int h = unit % H, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, C = H * kN;
    const i64 base = unit / H * T * C + h * kN;
    float wrong = 0.f;
    if (warp >= 4) {
        // ---- operands: channels 2 lane, 2 lane + 1 of four tokens ----------------------------------------------------------
        constexpr int R = 4;
        const int p = warp - 4, t0 = R * p, c = 2 * lane, tid = threadIdx.x - 128;
        const bool vec = vec_ok(a_, 2) && vec_ok(w_, 2), wide = sizeof(E) == 2 && vec_ok(b_, 8), vecb = vec_ok(b_, 2);
        struct Raw {   // of two segments: what is asked for in one step of the loop below is read two steps later
            Pair<E> aa[R], ww[STATIC ? 1 : R], bb[R];
            uint4 bw;
        } raw[2];
        auto fetch = [&](Raw& x, int it) {
            const int seg = REV ? nseg - 1 - it : it, n = min(kSeg, T - seg * kSeg);
            const i64 o = base + (i64)seg * kSeg * C;
            read_rows<E, R>(x.aa, a_ + o + c, t0, n, C, vec);
            if constexpr (!STATIC) read_rows<E, R>(x.ww, w_ + o + c, t0, n, C, vec);
            if (wide) {
                const int row = tid >> 3;
                x.bw = row < n ? __ldg(reinterpret_cast<const uint4*>(b_ + o + (i64)row * C + 8 * (tid & 7))) : make_uint4(0u, 0u, 0u, 0u);
            } else read_rows<E, R>(x.bb, b_ + o + c, t0, n, C, vecb);
            const int far = REV ? seg - 6 : seg + 6;   // (two steps are not long enough for HBM)
            if (far >= 0 && far < nseg && tid < (STATIC ? 64 : 96)) {
                const E* y = tid < 32 ? a_ : tid < 64 ? b_ : w_;
                prefetch_rows(y, base + (i64)far * kSeg * C, min(kSeg, T - far * kSeg), C, lane);
            }
        };
        if constexpr (STATIC) {
            raw[0].ww[0] = raw[1].ww[0] = read_pair(w_ + h * kN + c, vec);
            if (!REV && p == 7 && flags != nullptr) {
                const bool out = __any_sync(0xffffffffu, beyond(log2_decay_static(decode(raw[0].ww[0])), kStaticRange));
                for (int i = lane; i < nseg; i += 32) flags[unit * nseg + i] = out;
            }
        }
        if (nseg > 1) fetch(raw[0], 0);
        if (nseg > 2) fetch(raw[1], 1);
        auto make = [&](Raw& x, int it) {
            const int seg = REV ? nseg - 1 - it : it, n = min(kSeg, T - seg * kSeg);
            ChainSmem<E>& sm = buf[it & 1];
            if (it >= 2) bar_join<3>(it & 1);
            float2 d[STATIC ? 1 : R], before, after;   // sums of log2 decays before and behind these tokens
            if constexpr (STATIC) d[0] = log2_decay_static(decode(x.ww[0]));
            else {
                float2 s = make_float2(0.f, 0.f);
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    d[i] = t0 + i < n ? log2_decay(decode(x.ww[i])) : make_float2(0.f, 0.f);
                    s.x += d[i].x; s.y += d[i].y;
                }
                *reinterpret_cast<float2*>(sm.tot + p * kN + c) = s;
                asm volatile("bar.sync 5, 256;" ::: "memory");
                before = after = make_float2(0.f, 0.f);
#pragma unroll
                for (int i = 0; i < kSeg / R; ++i) {
                    const float2 t = *reinterpret_cast<const float2*>(sm.tot + i * kN + c);
                    if (i < p) { before.x += t.x; before.y += t.y; }
                    if (i > p) { after.x += t.x; after.y += t.y; }
                }
                if (p == 0) *reinterpret_cast<float2*>(sm.f + c) = make_float2(ex2(s.x + after.x), ex2(s.y + after.y));
            }
            if (STATIC && p == 0) {   // (exact to a rounding: the same factor acts once per segment)
                const float2 w = decode(x.ww[0]);
                *reinterpret_cast<float2*>(sm.f + c) = make_float2(expf(-expf(w.x) * n), expf(-expf(w.y) * n));
            }
#pragma unroll
            for (int j = 0; j < R; ++j) {
                const int i = REV ? j : R - 1 - j;   // towards the end that the products count from, starting there
                const float2 a = decode(x.aa[i]);
                float2 e;
                if constexpr (STATIC) {
                    const int m = REV ? t0 + i : max(n - 1 - (t0 + i), 0);
                    e = m == 0 ? make_float2(0.f, 0.f) : make_float2(d[0].x * m, d[0].y * m);   // (also for a decay of 0, whose logarithm is -inf)
                } else {
                    float2& s = REV ? before : after;
                    e = s;
                    s.x += d[i].x; s.y += d[i].y;
                }
                put_split(sm.A, t0 + i, lane, a.x * ex2(e.x), a.y * ex2(e.y));
            }
            if (wide) {
                put_eight(sm.B, tid >> 3, tid & 7, x.bw);
            } else {
#pragma unroll
                for (int i = 0; i < R; ++i) put_pair<E>(sm.B, t0 + i, lane, x.bb[i]);
            }
            if (it + 3 < nseg) fetch(x, it + 2);
            bar_tell<1>(it & 1);
        };
        for (int it = 0; it + 1 < nseg; it += 2) {
            make(raw[0], it);
            if (it + 2 < nseg) make(raw[1], it + 1);
        }
    } else {
        // ---- the state: keys 16 warp + at16(g), + 2 of all values -----------------------------------------------------------------------
        const int g = lane >> 2, q = lane & 3;
        const uint32_t fa = frag_cols(0, 2 * warp, lane), fb = frag_rows(0, 0, lane);   // (an even piece further on: XOR, see img_at)
        float s[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[i][e] = 0.f;
        for (int it = 0; it < nseg; ++it) {
            float* p = states + (unit * nseg + (REV ? nseg - 1 - it : it)) * kN * kN + (16 * warp + at16(g)) * kN + 4 * q;
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    *reinterpret_cast<float4*>(p + 2 * e * kN + 16 * i) = make_float4(s[2 * i][2 * e], s[2 * i][2 * e + 1], s[2 * i + 1][2 * e], s[2 * i + 1][2 * e + 1]);
            if (it + 1 == nseg) break;
            bar_join<1>(it & 1);
            const ChainSmem<E>& sm = buf[it & 1];
            const float f0 = sm.f[16 * warp + at16(g)], f1 = sm.f[16 * warp + at16(g) + 2];
            // The segment's own sums from zero, four side by side, then one rounded multiply-add per state element: the tensor core's sums are
            // cut off, not rounded, and with the state itself as the accumulator that adds up along the sequence.  Errors of the states in norm
            // (B2 T1000 H40; local sums and a scan in fp32 / state as accumulator / this): decay inputs around -10 6.4e-6 (there the rounding of
            // the decays themselves) / 2.3e-6 / 2.1e-7, -5 3.1e-7 / 3.9e-7 / 1.2e-7, -1 5.7e-8 / 6.5e-8 / 6.7e-8, 1 3.0e-8 / 5.0e-8 / 5.0e-8
            // (one cut of the newest tokens' sum).  B8 T1000 H32 497 -> 501 us.
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                float c[2][1][2][4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int e = 0; e < 4; ++e) c[i / 2][0][i & 1][e] = 0.f;
                if constexpr (NV == 1) {
                    uint32_t b[2][2][4];
#pragma unroll
                    for (int kt = 0; kt < 2; ++kt)
#pragma unroll
                        for (int i = 0; i < 2; ++i) ldsm_t(b[kt][i], smem_addr(sm.B) + 16 * kt * 128 + (fb ^ (4 * half + 2 * i) << 4));
#pragma unroll
                    for (int pa = 2; pa >= 0; --pa)   // the small parts of all tokens first: what is cut off behind them is small too
#pragma unroll
                        for (int kt = 0; kt < 2; ++kt) {
                            uint32_t a[4];
                            ldsm_t(a, smem_addr(sm.A) + pa * kImg + 16 * kt * 128 + fa);
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                mma(c[i][0][0], a, b[kt][i][0], b[kt][i][1]);
                                mma(c[i][0][1], a, b[kt][i][2], b[kt][i][3]);
                            }
                        }
                } else {
#pragma unroll
                    for (int kt = 0; kt < 2; ++kt) {
                        uint32_t a[1][3][4], b[2][NV][4];
                        ldsm_t<3>(a[0], smem_addr(sm.A) + 16 * kt * 128 + fa);
#pragma unroll
                        for (int i = 0; i < 2; ++i) ldsm_t<NV>(b[i], smem_addr(sm.B) + 16 * kt * 128 + (fb ^ (4 * half + 2 * i) << 4));
#pragma unroll
                        for (int i = 0; i < 2; ++i) mma_split<true, 1, 3, NV>(c[i], a, b[i]);
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int e = 0; e < 4; ++e) s[4 * half + i][e] = fmaf(s[4 * half + i][e], e < 2 ? f0 : f1, c[i / 2][0][i & 1][e]);
            }
            if (it + 3 < nseg) bar_tell<3>(it & 1);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {   // (what is not finite stays so: the last state tells)
            check(wrong, make_float2(s[i][0], s[i][1]));
            check(wrong, make_float2(s[i][2], s[i][3]));
        }
    }
    if (__syncthreads_or(wrong != 0.f)) walk_again<E, STATIC, REV>(T, nseg, C, a_ + base, b_ + base, w_ + (STATIC ? h * kN : base), states + unit * nseg * kN * kN);
}

// ---- the segments that the kernels above have left ----------------------------------------------------------------------------
// ONE: a block per segment (flags: none, or whether it is one of those).  Else block b looks at the segments b, b + grid, .. together: with
// none flagged, starting the blocks is all that the launch costs.
template <bool ONE, typename F>
__device__ __forceinline__ void for_flagged(const int* __restrict__ flags, i64 total, F body) {
    if constexpr (ONE) {
        if (flags == nullptr || flags[blockIdx.x]) body((i64)blockIdx.x);
    } else {
        __shared__ unsigned found[4];   // a bit per thread of up to 128
        for (i64 first = blockIdx.x; first < total; first += (i64)gridDim.x * blockDim.x) {
            const i64 mine = first + (i64)threadIdx.x * gridDim.x;
            const bool flag = mine < total && flags[mine];
            const unsigned bits = __ballot_sync(0xffffffffu, flag);
            if ((threadIdx.x & 31) == 0) found[threadIdx.x >> 5] = bits;
            if (!__syncthreads_or(flag)) continue;
            for (int w = 0; w < (int)blockDim.x / 32; ++w)
                for (unsigned left = found[w]; left != 0; left &= left - 1) {
                    body(first + (i64)(32 * w + __ffs(left) - 1) * gridDim.x);
                    __syncthreads();
                }
            __syncthreads();
        }
    }
}
// A block per segment up to eight rounds of resident blocks: nothing is faster where all are flagged.  Above, four rounds of blocks, because with
// none flagged it is the rounds that cost.  B8 T1000 H32, 8192 segments, y and gradients, none flagged / all: a block each 8 + 14 / 223 + 627 us,
// four rounds 6 + 6 / 277 + 684, one 4.5 + 4.3 / 301 + 694.
inline i64 resident_blocks(int per_sm) { return (i64)(sm_count() > 0 ? sm_count() : 148) * per_sm; }
inline bool block_per_segment(i64 total, int per_sm) { return total <= 8 * resident_blocks(per_sm); }

// ---- launches ----------------------------------------------------------------------------------------------------------------
// One block per unit walks all segments, or (the other kernels) every segment on its own and a scan: with few units the walk is
// as long as T, and the scan's passes over the states cost little.  Forward + backward, us, scan / walk: RWKV-6 T999 48 units 166 / 176, 64 units
// 205 / 204 (T4095 812 / 700), 80 units 255 / 227; RWKV-5 fp32 183 / 190, 226 / 221 (896 / 767), 275 / 253.
inline bool seg_chain_pays(i64 units) { return units * 2 > sm_count(); }
// Up to four segments per SM the token-by-token kernels take all of them: a launch less each way, and little to win.  Us, those / by
// products, RWKV-6 and RWKV-5 fp32: 256 segments 95 / 101 and 91 / 96, 384 102 / 100 and 99 / 96, 512 121 / 100 and 108 / 97 (one sequence), 90 / 93
// and 88 / 94 (eight of 100 tokens: 592 is where none is slower), 608 137 / 100 and 124 / 98, 768 149 / 103 and 138 / 108.  (About 90 us are the host's.)
inline bool seg_mma_pays(i64 total) { return total > 4ll * sm_count(); }

template <typename E, bool STATIC, bool REV>
int seg_chain(i64 units, int T, int H, int nseg, const void* a, const void* b, const void* w, float* states, int* flags, cudaStream_t st) {
    constexpr int smem = 2 * sizeof(ChainSmem<E>);
    const cudaError_t e = allow_smem<seg_mma_chain_kernel<E, STATIC, REV>>(smem);
    RWKV_REQUIRE(e == cudaSuccess, RWKVB200_ECUDA, "training on segments: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    seg_mma_chain_kernel<E, STATIC, REV><<<(unsigned)units, 384, smem, st>>>(T, H, nseg, (const E*)a, (const E*)b, (const E*)w, states, flags);
    return check_launch("training on segments: states");
}
template <typename E, bool STATIC>
int seg_mma_y(i64 total, int T, int H, int nseg, const void* r, const void* k, const void* v, const void* w, const void* u, const float* states,
              void* y, int* flags, bool known, cudaStream_t st) {
    constexpr int smem = sizeof(YSmem<E>);
    const cudaError_t e = allow_smem<seg_mma_y_kernel<E, STATIC>>(smem);
    RWKV_REQUIRE(e == cudaSuccess, RWKVB200_ECUDA, "training on segments: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    seg_mma_y_kernel<E, STATIC><<<(unsigned)total, 128, smem, st>>>(T, H, nseg, (const E*)r, (const E*)k, (const E*)v, (const E*)w, (const E*)u, states,
                                                                   (E*)y, flags, known, 4 * sm_count());
    return check_launch("training on segments: y");
}
template <typename E, bool STATIC>
int seg_mma_backward(i64 total, int T, int H, int nseg, const void* r, const void* k, const void* v, const void* w, const void* u, const void* gy,
                     const float* S, const float* D, void* gr, void* gk, void* gv, void* gw, float* partial, const int* left, int* flags, cudaStream_t st) {
    constexpr int smem = sizeof(BwdSmemM<E>);
    const cudaError_t e = allow_smem<seg_mma_backward_kernel<E, STATIC>>(smem);
    RWKV_REQUIRE(e == cudaSuccess, RWKVB200_ECUDA, "training on segments: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    seg_mma_backward_kernel<E, STATIC><<<(unsigned)total, 128, smem, st>>>(T, H, nseg, (const E*)r, (const E*)k, (const E*)v, (const E*)w, (const E*)u,
                                                                          (const E*)gy, S, D, (E*)gr, (E*)gk, (E*)gv, (E*)gw, partial, left, flags,
                                                                          4 * sm_count());
    return check_launch("training on segments: gradients");
}

}  // namespace
}  // namespace rwkvb200
