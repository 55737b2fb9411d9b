// Pieces of the fp32 kernels that work on the time segments of a sequence at the same time (wkv5_seg.cu, wkv6_seg.cu): rows
// of a segment in shared memory, register tiles of a state, sums over lanes.
#pragma once
#include "packed.cuh"

namespace rwkvb200 {
namespace {

constexpr int kSeg = 32, kN = 64;   // tokens of a segment; head size of the tiles (smaller heads are padded with zeros)

// Rows of 64 channels in shared memory: the first four of every eight channels come first, then the other four, so that lanes
// that own eight channels each read 16-byte pieces without bank conflicts.
__device__ __forceinline__ int place(int ch) { return ((ch & 4) << 3) + ((ch >> 3) << 2) + (ch & 3); }
struct Eight { float4 lo, hi; };
__device__ __forceinline__ Eight load8(const float* row, int grp) {
    return Eight{*reinterpret_cast<const float4*>(row + 4 * grp), *reinterpret_cast<const float4*>(row + 32 + 4 * grp)};
}
__device__ __forceinline__ void pairs(const Eight& x, f2 (&p)[4]) {
    p[0] = pack2(x.lo.x, x.lo.y); p[1] = pack2(x.lo.z, x.lo.w); p[2] = pack2(x.hi.x, x.hi.y); p[3] = pack2(x.hi.z, x.hi.w);
}
__device__ __forceinline__ void twice(const Eight& x, f2 (&p)[8]) {
    p[0] = pack2(x.lo.x, x.lo.x); p[1] = pack2(x.lo.y, x.lo.y); p[2] = pack2(x.lo.z, x.lo.z); p[3] = pack2(x.lo.w, x.lo.w);
    p[4] = pack2(x.hi.x, x.hi.x); p[5] = pack2(x.hi.y, x.hi.y); p[6] = pack2(x.hi.z, x.hi.z); p[7] = pack2(x.hi.w, x.hi.w);
}

// Stages `n` tokens of a (T, C) tensor as fp32 rows, zero where there is no token or channel, each times scale(token, channel).
// Whole aligned heads are read four channels at a time with every load of the thread in flight.
__device__ __forceinline__ float4 read4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 read4(const bf16* p) {
    const uint2 x = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(x.x << 16), __uint_as_float(x.x & 0xffff0000u), __uint_as_float(x.y << 16), __uint_as_float(x.y & 0xffff0000u));
}
template <int NTH, typename E, typename F>
__device__ __forceinline__ void stage(float* dst, const E* __restrict__ src, int n, int C, int N, int tid, F scale) {
    if (N == kN && (reinterpret_cast<uintptr_t>(src) & (4 * sizeof(E) - 1)) == 0) {
        constexpr int PER = kSeg * kN / 4 / NTH;
        float4 x[PER];
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int t = (i * NTH + tid) / 16, j = (tid & 15) * 4;
            x[i] = t < n ? read4(src + (i64)t * C + j) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int t = (i * NTH + tid) / 16, j = (tid & 15) * 4;
            *reinterpret_cast<float4*>(dst + t * kN + place(j)) =
                make_float4(x[i].x * scale(t, j), x[i].y * scale(t, j + 1), x[i].z * scale(t, j + 2), x[i].w * scale(t, j + 3));
        }
    } else {
        for (int x = tid; x < kSeg * kN; x += NTH) {
            const int t = x / kN, j = x % kN;
            dst[t * kN + place(j)] = (t < n && j < N) ? to_f(src[(i64)t * C + j]) * scale(t, j) : 0.f;
        }
    }
}
template <int NTH, typename E>
__device__ __forceinline__ void stage(float* dst, const E* __restrict__ src, int n, int C, int N, int tid) {
    stage<NTH>(dst, src, n, C, N, tid, [](int, int) { return 1.f; });
}

// A lane's tile of a state, x[value][key pair]: 8 values from v0 on, 8 keys from k0 on; states are [key][value] in memory.
typedef f2 Tile[8][4];
// key pair p of the tile
__device__ __forceinline__ void load_pair(f2 (&x)[8], int p, const float* st, int k0, int v0, int N) {
    float a[2][8];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const float* row = st + (i64)(k0 + 2 * p + e) * N + v0;
        if (N == kN) {
            *reinterpret_cast<float4*>(a[e]) = *reinterpret_cast<const float4*>(row);
            *reinterpret_cast<float4*>(a[e] + 4) = *reinterpret_cast<const float4*>(row + 4);
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) a[e][i] = (k0 + 2 * p + e < N && v0 + i < N) ? row[i] : 0.f;
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = pack2(a[0][i], a[1][i]);
}
__device__ __forceinline__ void load_tile(Tile& x, const float* st, int k0, int v0, int N) {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        f2 q[8];
        load_pair(q, p, st, k0, v0, N);
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i][p] = q[i];
    }
}
__device__ __forceinline__ void store_tile(const Tile& x, float* st, int k0, int v0, int N) {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        float a[2][8];
#pragma unroll
        for (int i = 0; i < 8; ++i) unpack2(x[i][p], a[0][i], a[1][i]);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            float* row = st + (i64)(k0 + 2 * p + e) * N + v0;
            if (N == kN) {
                *reinterpret_cast<float4*>(row) = *reinterpret_cast<const float4*>(a[e]);
                *reinterpret_cast<float4*>(row + 4) = *reinterpret_cast<const float4*>(a[e] + 4);
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (k0 + 2 * p + e < N && v0 + i < N) row[i] = a[e][i];
            }
        }
    }
}

// Sums of v[0..7] over the 8 lanes that differ in bits 2 to 4, in 7 shuffles: a lane ends with element (lane >> 2) of them.
__device__ __forceinline__ float reduce8(float (&v)[8], int lane) {
#pragma unroll
    for (int m = 16, n = 4; n >= 1; m >>= 1, n >>= 1) {
        const bool up = (lane & m) != 0;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
        }
    }
    return v[0];
}
// The same over the 4 lanes that differ in bits 0 and 1: a lane ends with elements 2 (lane & 3) and the next, in v[0], v[1].
__device__ __forceinline__ void reduce8_pairs(float (&v)[8], int lane) {
#pragma unroll
    for (int m = 2, n = 4; n >= 2; m >>= 1, n >>= 1) {
        const bool up = (lane & m) != 0;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
        }
    }
}

}  // namespace
}  // namespace rwkvb200
