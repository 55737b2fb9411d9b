// depthwise_conv1d by Fourier transforms (timex_fft.cu).
#pragma once
#include "common.cuh"

namespace rwkvb200 {

constexpr int kTimexSplits = 8;   // most parts of the batch that the backward works on at the same time
bool timex_fft_applies(int T);
int timex_fft_forward(const float* w, const float* k, float* x, float eps, int B, int C, int T, cudaStream_t st);
// gw (C,T): summed over the batch.  work: kTimexSplits * C * T floats, or NULL (then the batch is not split).
int timex_fft_backward(const float* w, const float* k, const float* g, float* gw, float* gk, float* work, int B, int C, int T, cudaStream_t st);

}  // namespace rwkvb200
