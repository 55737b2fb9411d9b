// RWKV-6 training in fp32 arithmetic, split over time: bf16, head size 64, no state in or out (wkv6_seg.cu).
#pragma once
#include "common.cuh"

namespace rwkvb200 {

// Which calls: a T that is not whole 16-token tiles, which the tensor-core kernels do not take.  Up to 32 tokens there is one
// segment, and the general-shape kernels have less to do.
inline bool wkv6_seg_applies(int dtype, int T, int N, bool state) { return dtype == RWKVB200_BF16 && N == 64 && !state && T > 32 && T % 16 != 0; }

// Floats of the buffer that the forward leaves for the backward: a state, the decays and a flag of every segment.
inline size_t wkv6_seg_saved(int B, int T, int H) { return (size_t)B * H * ((T + 31) / 32) * (64 * 64 + 64 + 1); }
// Floats of the backward's work buffer: an adjoint state per segment; (B * segments, C) partials of gu and a flag per segment come
// behind it.
inline size_t wkv6_seg_adjoints(int B, int T, int C) { return (size_t)B * ((T + 31) / 32) * C * 64; }
inline size_t wkv6_seg_flags(int B, int T, int C) { return (size_t)B * ((T + 31) / 32) * (C / 64); }
inline long long wkv6_seg_rows(int B, int T) { return (long long)B * ((T + 31) / 32); }

// w: raw decay input (B,T,C), bf16 like r, k, v, u (H,N), gy and the outputs.
int wkv6_seg_forward(int B, int T, int H, const void* r, const void* k, const void* v, const void* w, const void* u, void* y, float* saved,
                     cudaStream_t st);
int wkv6_seg_backward(int B, int T, int H, const void* r, const void* k, const void* v, const void* w, const void* u, const void* gy, void* gr,
                      void* gk, void* gv, void* gw, const float* saved, float* adjoints, float* gu_partial, int* flags, cudaStream_t st);

}  // namespace rwkvb200
