// RWKV-5 training in fp32 arithmetic, split over time (wkv5_seg.cu).
#pragma once
#include "common.cuh"

namespace rwkvb200 {

constexpr int kWkv5Seg = 32;   // tokens of a segment
inline size_t wkv5_seg_count(int T) { return (size_t)(T + kWkv5Seg - 1) / kWkv5Seg; }

// w: raw decay input (H,N) in the activation type.  states: (B,H,segments,N,N) fp32, left for the backward (its S).
int wkv5_seg_forward(int dtype, int B, int T, int C, int H, const void* r, const void* k, const void* v, const void* w, const void* u, void* y,
                     float* states, int* flags, cudaStream_t st);
// left: the forward's flags.  D: work of the size of `states`.  partial: (B * segments, 2, C) fp32, the gradients of w and u of every segment.
int wkv5_seg_backward(int dtype, int B, int T, int C, int H, const void* r, const void* k, const void* v, const void* w, const void* u,
                      const void* gy, void* gr, void* gk, void* gv, const float* S, float* D, float* partial, const int* left, int* flags, cudaStream_t st);

}  // namespace rwkvb200
