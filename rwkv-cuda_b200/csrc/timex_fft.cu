// depthwise_conv1d by Fourier transforms, fp32: the three correlations of timex.cu are causal convolutions of length T,
//   x[t]  = eps + sum_{u<=t} w'[t-u] k[u]      gk'[t] = sum_{u<=t} w'[t-u] g'[u]      gw[t] = sum_b sum_{u<=t} g'_b[t-u] k_b[u]
// with w'[j] = w[T-1-j] and so on (index reversed).  The direct form does T/2 multiply-adds per element on the FP32 pipe
// (T = 768: 43.5 GFLOP forward + backward at B32 C768, 584 us at the nominal peak, 1365 us measured); transforms of length
// N >= 2 T do about 20 log2(N) operations per element, a sixth of that at T = 768, still entirely in fp32.
//
// Two batch rows are the real and the imaginary part of one complex row: the filter is real, so the convolution of
// k1 + i k2 is x1 + i x2.  For gw the rows of g are packed as g1 - i g2: (K1 + i K2)(G1 - i G2) has the spectrum of
// k1*g1 + k2*g2 as its real sequence, so products are summed over the batch and transformed back once.
//
// The rounding of a transform is relative to the norm of what goes into it.  Rows whose norms differ are therefore not packed
// together (a small row would carry the large one's rounding, a row of zeros would come back as noise): they are done one after
// the other.  A value that is not finite, or too large for the sums of a transform, would spoil the whole row, the tokens before
// it too, and the row beside it: such a row, and all rows of a channel whose filter has such a value, are added up directly.
// What remains is a bound by row: errors are about 4 2^-24 of (norm of the filter) x (norm of the row), at early tokens too.
//
// A transform of N = 256 R points (R = 4, 6, 8) is done by N/16 threads with 16 points each: radix 16, exchange through shared
// memory, radix 16, exchange inside groups of R threads, radix R (6 does not divide 16: two of the six threads of a
// group leave a third of that step idle, 18 places for 16 points).  Spectra stay in the order this leaves them in (thread and
// register); the inverse takes the same steps backwards, so nothing is ever reordered.  The upper half of the input is zero
// and the upper half of the output is not needed: the outer radix-16 steps do half of their work.  Row strides in shared
// memory (L + R, and 16 (R+1) + R) make every exchange conflict free.  128 threads per block, 2048 / N transforms at
// a time (1536 points: 96 threads, one).
// B32 C768 T768 on a B200: forward 357 us direct, 112 us with 2048 points, 102 us with 1536; backward with its gw over the batch 1017,
// 218 and 182 us (compiled for three blocks of 96 threads per SM; for four 191; looking at the pairs took 19 us of these with a
// barrier of its own, 2 or 3 less with the vote at the first barrier of a transform), and 5 us to
// sum its parts.
// Errors against fp64 are 2.4e-7 of the norm (direct: 4.1e-7).
#include "timex_fft.cuh"

namespace rwkvb200 {
namespace {

struct cf { float x, y; };
__device__ __forceinline__ cf operator+(cf a, cf b) { return cf{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ cf operator-(cf a, cf b) { return cf{a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ cf mul(cf a, cf b) { return cf{fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x)}; }
__device__ __forceinline__ cf mulc(cf a, cf b) { return cf{fmaf(a.x, b.x, a.y * b.y), fmaf(a.y, b.x, -a.x * b.y)}; }   // a conj(b)
template <bool INV> __device__ __forceinline__ cf tw(cf a, cf b) { return INV ? mulc(a, b) : mul(a, b); }
// a times -i (forward) or i (inverse)
template <bool INV> __device__ __forceinline__ cf quarter(cf a) { return INV ? cf{-a.y, a.x} : cf{a.y, -a.x}; }

// natural order in and out
template <bool INV>
__device__ __forceinline__ void fft4(cf& a, cf& b, cf& c, cf& d) {
    const cf s = a + c, e = a - c, p = b + d, q = quarter<INV>(b - d);
    a = s + p; c = s - p; b = e + q; d = e - q;
}
// the same when the inputs c and d are zero
template <bool INV>
__device__ __forceinline__ void fft4_half(cf& a, cf& b, cf& c, cf& d) {
    const cf q = quarter<INV>(b);
    c = a - b; d = a - q; const cf t = a + q; a = a + b; b = t;
}
template <bool INV>
__device__ __forceinline__ void fft3(cf& a, cf& b, cf& c) {
    constexpr float h = 0.86602540378443865f;
    const cf s = b + c, d = quarter<INV>(cf{h * (b.x - c.x), h * (b.y - c.y)}), m = cf{fmaf(-0.5f, s.x, a.x), fmaf(-0.5f, s.y, a.y)};
    a = a + s; b = m + d; c = m - d;
}
template <bool INV>
__device__ __forceinline__ void fft6(cf (&v)[6]) {   // two of length 3, W6^k = exp(-2 pi i k / 6) on the odd one
    constexpr float h = 0.86602540378443865f;
    fft3<INV>(v[0], v[2], v[4]);
    fft3<INV>(v[1], v[3], v[5]);
    const cf e0 = v[0], e1 = v[2], e2 = v[4], o0 = v[1], o1 = tw<INV>(v[3], cf{0.5f, -h}), o2 = tw<INV>(v[5], cf{-0.5f, -h});
    v[0] = e0 + o0; v[3] = e0 - o0; v[1] = e1 + o1; v[4] = e1 - o1; v[2] = e2 + o2; v[5] = e2 - o2;
}
template <bool INV>
__device__ __forceinline__ void fft8(cf (&v)[8]) {
    constexpr float h = 0.70710678118654752f;
    fft4<INV>(v[0], v[2], v[4], v[6]);
    fft4<INV>(v[1], v[3], v[5], v[7]);
    // odd half: v[1], v[3], v[5], v[7] hold its outputs 0..3; twiddles W8^k
    const cf o1 = tw<INV>(v[3], cf{h, -h}), o2 = quarter<INV>(v[5]), o3 = tw<INV>(v[7], cf{-h, -h}), o0 = v[1];
    const cf e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    v[0] = e0 + o0; v[4] = e0 - o0; v[1] = e1 + o1; v[5] = e1 - o1;
    v[2] = e2 + o2; v[6] = e2 - o2; v[3] = e3 + o3; v[7] = e3 - o3;
}
// radix 16 as 4 x 4, natural order in and out; HALF: inputs 8..15 are zero (and not read)
template <bool INV, bool HALF, int V>
__device__ __forceinline__ void fft16(cf (&v)[V]) {
    constexpr float c1 = 0.92387953251128674f, s1 = 0.38268343236508977f, h = 0.70710678118654752f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (HALF) fft4_half<INV>(v[i], v[i + 4], v[i + 8], v[i + 12]);
        else fft4<INV>(v[i], v[i + 4], v[i + 8], v[i + 12]);
    }
    v[5] = tw<INV>(v[5], cf{c1, -s1});
    v[6] = tw<INV>(v[6], cf{h, -h});
    v[7] = tw<INV>(v[7], cf{s1, -c1});
    v[9] = tw<INV>(v[9], cf{h, -h});
    v[10] = quarter<INV>(v[10]);
    v[11] = tw<INV>(v[11], cf{-h, -h});
    v[13] = tw<INV>(v[13], cf{s1, -c1});
    v[14] = tw<INV>(v[14], cf{-h, -h});
    v[15] = tw<INV>(v[15], cf{-c1, s1});
    cf t[16];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        fft4<INV>(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
#pragma unroll
        for (int q = 0; q < 4; ++q) t[k + 4 * q] = v[4 * k + q];
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = t[k];
}

template <int R>
struct Plan {
    static constexpr int N = 256 * R, L = 16 * R, kThreads = R % 3 ? 128 : 96, G = kThreads / L;   // length, threads per transform, transforms at a time
    static constexpr int E = (16 + R - 1) / R, V = R * E;             // transforms of length R per thread, their points
    static constexpr int S1 = L + R, P2 = R + 1, S2 = 16 * P2 + R;    // strides of the two exchanges
    static constexpr int kBuf1 = 16 * S1, kBuf2 = 16 * S2;            // complex numbers per transform
    static constexpr int kRatio = R <= 4 ? 2 : 3;   // see apart()
    static constexpr int kSmem = (G * (kBuf1 + kBuf2) + V * L) * sizeof(cf);
};

// Powers 1, 2, 4, 8 of a thread's twiddle; the other eleven are products of these.
struct Twiddles {
    cf w1, w2, w4, w8;
    __device__ __forceinline__ void set(float turns) {   // exp(-2 pi i turns) and its powers
        cf* p[4] = {&w1, &w2, &w4, &w8};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float s, c;
            sincospif(2.f * turns * (float)(1 << i), &s, &c);
            *p[i] = cf{c, -s};
        }
    }
    template <bool INV, int V>
    __device__ __forceinline__ void apply(cf (&v)[V]) const {
        v[1] = tw<INV>(v[1], w1); v[2] = tw<INV>(v[2], w2); v[4] = tw<INV>(v[4], w4); v[8] = tw<INV>(v[8], w8);
        const cf w3 = mul(w1, w2);
        v[3] = tw<INV>(v[3], w3);
        v[5] = tw<INV>(v[5], mul(w1, w4)); v[6] = tw<INV>(v[6], mul(w2, w4)); v[7] = tw<INV>(v[7], mul(w3, w4));
        v[9] = tw<INV>(v[9], mul(w1, w8)); v[10] = tw<INV>(v[10], mul(w2, w8)); v[11] = tw<INV>(v[11], mul(w3, w8));
        const cf w12 = mul(w4, w8);
        v[12] = tw<INV>(v[12], w12);
        v[13] = tw<INV>(v[13], mul(w1, w12)); v[14] = tw<INV>(v[14], mul(w2, w12)); v[15] = tw<INV>(v[15], mul(w3, w12));
    }
};

template <int R>
struct Engine {
    using P = Plan<R>;
    cf *b1, *b2;         // this transform's exchange buffers
    int j, k1, j1;
    Twiddles t1, t2;
    __device__ __forceinline__ Engine(cf* smem, int tid) {
        const int g = tid / P::L;
        j = tid % P::L; k1 = j / R; j1 = j % R;
        b1 = smem + g * P::kBuf1;
        b2 = smem + P::G * P::kBuf1 + g * P::kBuf2;
        t1.set((float)j / P::N);
        t2.set((float)j1 / P::L);
    }
    static constexpr int V = P::V;
    static __device__ __forceinline__ void group_sync() {   // groups of 6 threads are not inside a warp
        if (R % 3) __syncwarp();
        else __syncthreads();
    }
    template <bool INV>
    static __device__ __forceinline__ void small(cf (&v)[V]) {   // this thread's transforms of length R
#pragma unroll
        for (int e = 0; e < P::E; ++e) {
            if constexpr (R == 4) fft4<INV>(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]);
            else {
                cf u[R];
#pragma unroll
                for (int i = 0; i < R; ++i) u[i] = v[R * e + i];
                if constexpr (R == 6) fft6<INV>(u);
                else fft8<INV>(u);
#pragma unroll
                for (int i = 0; i < R; ++i) v[R * e + i] = u[i];
            }
        }
    }
    // v[m] = element j + L m (m < 8) -> spectrum.  A forward right after another forward needs a __syncthreads before it (the
    // other threads may still read the first exchange); between forward and inverse every thread writes what only it has read.
    // VOTE: the block's first barrier also asks whether any thread is against it; if so, nothing more is done and the answer is true.
    template <bool VOTE>
    __device__ __forceinline__ bool forward(cf (&v)[V], bool against) {
        fft16<false, true>(v);
        t1.apply<false>(v);
#pragma unroll
        for (int k = 0; k < 16; ++k) b1[k * P::S1 + j] = v[k];
        if (VOTE) { if (__syncthreads_or(against)) return true; }
        else __syncthreads();
#pragma unroll
        for (int m = 0; m < 16; ++m) v[m] = b1[k1 * P::S1 + j1 + R * m];
        fft16<false, false>(v);
        t2.apply<false>(v);
        group_sync();
#pragma unroll
        for (int k = 0; k < 16; ++k) b2[k1 * P::S2 + k * P::P2 + j1] = v[k];
        group_sync();
#pragma unroll
        for (int e = 0; e < P::E; ++e)
#pragma unroll
            for (int i = 0; i < R; ++i) v[e * R + i] = 16 % R == 0 || j1 + R * e < 16 ? b2[k1 * P::S2 + (j1 + R * e) * P::P2 + i] : cf{0.f, 0.f};
        small<false>(v);
        return false;
    }
    __device__ __forceinline__ void forward(cf (&v)[V]) { forward<false>(v, false); }
    // spectrum -> elements j + L m in v[m] (m < 8 are what the callers use), times N
    __device__ __forceinline__ void inverse(cf (&v)[V]) {
        small<true>(v);
        group_sync();
#pragma unroll
        for (int e = 0; e < P::E; ++e)
            if (16 % R == 0 || j1 + R * e < 16)
#pragma unroll
                for (int i = 0; i < R; ++i) b2[k1 * P::S2 + (j1 + R * e) * P::P2 + i] = v[e * R + i];
        group_sync();
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = b2[k1 * P::S2 + k * P::P2 + j1];
        t2.apply<true>(v);
        fft16<true, false>(v);
#pragma unroll
        for (int m = 0; m < 16; ++m) b1[k1 * P::S1 + j1 + R * m] = v[m];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = b1[k * P::S1 + j];
        t1.apply<true>(v);
        fft16<true, false>(v);
    }
};

// Values up to this size cannot overflow in a transform, in the product of two spectra or in its sum over the batch.
constexpr float kLargest = 1e15f;
__device__ __forceinline__ bool unfit(float x) { return !(fabsf(x) <= kLargest); }   // NaN and infinities too

// A row alone (this thread has 8 elements of it): has it one?
template <int V>
__device__ __forceinline__ bool unfit(const cf (&v)[V]) {
    bool u = false;
#pragma unroll
    for (int m = 0; m < 8; ++m) u |= unfit(v[m].x);
    return u;
}

// Whether the two rows of v must not be packed (this thread has 8 elements of each): true in some thread of the block if the
// sums of squares of a warp's elements differ by more than RATIO, are too small to compare, or so large that an element may be
// unfit.  Rounding of the smaller row grows by sqrt((1 + RATIO) / 2) at most: with 2 up to 512 tokens and 3 above, packed rows
// stay about as exact as the direct sum (2.6e-7 at T = 257, where that has 2.4e-7; 3.3e-7 at 513, as that).
// `both`: there is a second row.
template <int RATIO, int V>
__device__ __forceinline__ bool apart(const cf (&v)[V], bool both, int lane) {
    float a = 0.f, b = 0.f;
    unsigned bits = 0;
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        a = fmaf(v[m].x, v[m].x, a);
        b = fmaf(v[m].y, v[m].y, b);
        bits |= __float_as_uint(v[m].x) | __float_as_uint(v[m].y);
    }
    const bool odd = !(a + b <= kLargest * kLargest) || (a + b < 1e-30f && (bits << 1) != 0);
    // the sums over the warp of RATIO a - b and RATIO b - a, each in half of the lanes
    const bool up = (lane & 16) != 0;
    const float d0 = fmaf((float)RATIO, a, -b), d1 = fmaf((float)RATIO, b, -a);
    float d = (up ? d1 : d0) + __shfl_xor_sync(0xffffffffu, up ? d0 : d1, 16);
#pragma unroll
    for (int m = 8; m >= 1; m >>= 1) d += __shfl_xor_sync(0xffffffffu, d, m);
    return odd || (both && !(d >= 0.f));
}

// out[t] = (add ? out[t] : eps) + sum_{u<=t} f[T-1-(t-u)] s[u] by the whole block; rev: s and out are indexed from the end
__device__ __noinline__ void direct(const float* f, const float* s, float* out, int T, bool rev, bool add, float eps) {
    for (int t = threadIdx.x; t < T; t += blockDim.x) {
        float acc = 0.f;
        for (int u = 0; u <= t; ++u) acc = fmaf(f[T - 1 - t + u], s[rev ? T - 1 - u : u], acc);
        float* p = out + (rev ? T - 1 - t : t);
        *p = acc + (add ? *p : eps);
    }
}

// spectrum of w' / N into shared memory, in the engine's order (Plan::V per thread of a transform); true if a value is unfit for it
template <int R>
__device__ __forceinline__ bool filter_spectrum(Engine<R>& fft, cf* Wh, const float* __restrict__ w, int T) {
    using P = Plan<R>;
    cf v[P::V];
    bool bad = false;
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        const int t = fft.j + P::L * m;
        v[m] = cf{t < T ? w[T - 1 - t] : 0.f, 0.f};
        bad |= unfit(v[m].x);
    }
    fft.forward(v);
    if (threadIdx.x < P::L)
#pragma unroll
        for (int k = 0; k < P::V; ++k) Wh[k * P::L + fft.j] = cf{v[k].x * (1.f / P::N), v[k].y * (1.f / P::N)};
    return __syncthreads_or(bad);
}

// What a transform works on in a pass: a pair of rows together, or its first and then its second row alone (as slot 0).
enum Pass { kTogether, kFirst, kSecond };

// grid (C, splits of the pairs of batch rows)
template <int R>
__global__ void __launch_bounds__(Plan<R>::kThreads, R % 3 ? 4 : 5) timex_fft_forward_kernel(const float* __restrict__ w, const float* __restrict__ k_,
                                                                        float* __restrict__ x_, float eps, int B, int C, int T) {
    using P = Plan<R>;
    extern __shared__ cf smem_fft[];
    __shared__ int bad[2 * P::G];   // rows that are added up directly
    cf* Wh = smem_fft + P::G * (P::kBuf1 + P::kBuf2);
    Engine<R> fft(smem_fft, threadIdx.x);
    const int c = blockIdx.x, pairs = (B + 1) / 2, g = threadIdx.x / P::L;
    if (threadIdx.x < 2 * P::G) bad[threadIdx.x] = 0;
    const bool bad_filter = filter_spectrum<R>(fft, Wh, w + (i64)c * T, T);
    Pass pass = kTogether;
    for (int p0 = blockIdx.y * P::G; p0 < pairs;) {
        const int b = 2 * (p0 + g) + (pass == kSecond);
        const i64 r0 = ((i64)b * C + c) * T, r1 = r0 + (i64)C * T;
        const int n0 = b < B ? T : 0, n1 = b + 1 < B && pass == kTogether ? T : 0;   // tokens of the two slots
        cf v[P::V];
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int t = fft.j + P::L * m;
            v[m] = cf{t < n0 ? k_[r0 + t] : 0.f, t < n1 ? k_[r1 + t] : 0.f};
        }
        const bool together = pass == kTogether;
        if (!together && (bad_filter || unfit(v))) bad[2 * g + (pass == kSecond)] = 1;
        if (fft.template forward<true>(v, together && (apart<P::kRatio>(v, n1 != 0, threadIdx.x & 31) || bad_filter))) { pass = kFirst; continue; }
#pragma unroll
        for (int k = 0; k < P::V; ++k) v[k] = mul(v[k], Wh[k * P::L + fft.j]);
        fft.inverse(v);
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int t = fft.j + P::L * m;
            if (t < n0) x_[r0 + t] = v[m].x + eps;
            if (t < n1) x_[r1 + t] = v[m].y + eps;
        }
        if (pass == kFirst) { pass = kSecond; continue; }
        if (pass == kSecond) {
            __syncthreads();
            for (int q = 0; q < 2 * P::G; ++q) {
                const int row = 2 * p0 + q;
                const i64 o = ((i64)row * C + c) * T;
                if (bad[q] && row < B) direct(w + (i64)c * T, k_ + o, x_ + o, T, false, false, eps);
            }
            __syncthreads();
            if (threadIdx.x < 2 * P::G) bad[threadIdx.x] = 0;
            __syncthreads();
            pass = kTogether;
        }
        p0 += gridDim.y * P::G;
    }
}

// gk, and the filter gradient summed over the batch rows of the block: gw[blockIdx.y][c][t]
template <int R>
__global__ void __launch_bounds__(Plan<R>::kThreads, 3) timex_fft_backward_kernel(const float* __restrict__ w, const float* __restrict__ k_,
                                                                         const float* __restrict__ g_, float* __restrict__ gw_,
                                                                         float* __restrict__ gk_, int B, int C, int T) {
    using P = Plan<R>;
    extern __shared__ cf smem_fft[];
    __shared__ int bad[2 * P::G];                 // rows that are added up directly
    __shared__ float gw_direct[8 * P::L];         // their part of gw
    cf* Wh = smem_fft + P::G * (P::kBuf1 + P::kBuf2);
    Engine<R> fft(smem_fft, threadIdx.x);
    const int c = blockIdx.x, pairs = (B + 1) / 2, g = threadIdx.x / P::L;
    if (threadIdx.x < 2 * P::G) bad[threadIdx.x] = 0;
    for (int t = threadIdx.x; t < 8 * P::L; t += P::kThreads) gw_direct[t] = 0.f;
    const bool bad_filter = filter_spectrum<R>(fft, Wh, w + (i64)c * T, T);
    cf acc[P::V];
#pragma unroll
    for (int k = 0; k < P::V; ++k) acc[k] = cf{0.f, 0.f};
    Pass pass = kTogether;
    for (int p0 = blockIdx.y * P::G; p0 < pairs;) {
        const int b = 2 * (p0 + g) + (pass == kSecond);
        const i64 r0 = ((i64)b * C + c) * T, r1 = r0 + (i64)C * T;
        const int n0 = b < B ? T : 0, n1 = b + 1 < B && pass == kTogether ? T : 0;
        cf z[P::V], v[P::V];
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int t = fft.j + P::L * m;
            z[m] = cf{t < n0 ? k_[r0 + t] : 0.f, t < n1 ? k_[r1 + t] : 0.f};
            v[m] = cf{t < n0 ? g_[r0 + T - 1 - t] : 0.f, t < n1 ? -g_[r1 + T - 1 - t] : 0.f};
        }
        bool against = false;
        if (pass == kTogether) {
            const bool za = apart<P::kRatio>(z, n1 != 0, threadIdx.x & 31), va = apart<P::kRatio>(v, n1 != 0, threadIdx.x & 31);
            against = za || va || bad_filter;
        } else if (unfit(z) || unfit(v)) {
            bad[2 * g + (pass == kSecond)] = 1;
        }
        if (fft.template forward<true>(z, against)) { pass = kFirst; continue; }
        __syncthreads();
        const bool skip = pass != kTogether && bad[2 * g + (pass == kSecond)];
        fft.forward(v);
#pragma unroll
        for (int k = 0; k < P::V; ++k) {
            if (!skip) acc[k] = acc[k] + mul(z[k], v[k]);
            v[k] = mul(v[k], Wh[k * P::L + fft.j]);
        }
        fft.inverse(v);
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int t = fft.j + P::L * m;
            if (t < n0) gk_[r0 + T - 1 - t] = v[m].x;
            if (t < n1) gk_[r1 + T - 1 - t] = -v[m].y;
        }
        if (pass == kFirst) { pass = kSecond; continue; }
        if (pass == kSecond) {
            __syncthreads();
            for (int q = 0; q < 2 * P::G; ++q) {
                const int row = 2 * p0 + q;
                const i64 o = ((i64)row * C + c) * T;
                if ((bad[q] || bad_filter) && row < B) direct(w + (i64)c * T, g_ + o, gk_ + o, T, true, false, 0.f);
                if (bad[q] && row < B) direct(g_ + o, k_ + o, gw_direct, T, false, true, 0.f);
            }
            __syncthreads();
            if (threadIdx.x < 2 * P::G) bad[threadIdx.x] = 0;
            __syncthreads();
            pass = kTogether;
        }
        p0 += gridDim.y * P::G;
    }
    // the spectra of the block's transforms are added up (each thread's points meet their likes at the same j), then one inverse
    __syncthreads();
    if (P::G > 1) {
        cf* sum = smem_fft;   // [G][V][L]
#pragma unroll
        for (int k = 0; k < P::V; ++k) sum[(g * P::V + k) * P::L + fft.j] = acc[k];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < P::V; ++k) {
            acc[k] = sum[k * P::L + fft.j];
#pragma unroll
            for (int q = 1; q < P::G; ++q) acc[k] = acc[k] + sum[(q * P::V + k) * P::L + fft.j];
        }
        __syncthreads();
    }
    fft.inverse(acc);
    if (g == 0)
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int t = fft.j + P::L * m;
            if (t < T) gw_[((i64)blockIdx.y * C + c) * T + t] = fmaf(acc[m].x, 1.f / P::N, gw_direct[t]);
        }
}

// Splits of the batch: enough blocks for four waves of the SMs' four blocks, but at least four rounds of pairs per block (the
// spectrum of the filter is made once per block).
int splits(int B, int C, int G, int most) {
    const int rounds = ((B + 1) / 2 + G - 1) / G;
    const int sms = sm_count();
    int s = 1;
    while (s < most && s * 2 <= rounds && (rounds / (s * 2) >= 4 || C * s < 4 * sms) && C * s < 16 * sms) s *= 2;
    return s;
}

template <int R>
int forward(const float* w, const float* k, float* x, float eps, int B, int C, int T, cudaStream_t st) {
    const cudaError_t e = allow_smem<timex_fft_forward_kernel<R>>(Plan<R>::kSmem);
    RWKV_REQUIRE(e == cudaSuccess, RWKVB200_ECUDA, "timex_forward: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    timex_fft_forward_kernel<R><<<dim3(C, splits(B, C, Plan<R>::G, 1 << 20)), Plan<R>::kThreads, Plan<R>::kSmem, st>>>(w, k, x, eps, B, C, T);
    return check_launch("timex_forward(transforms)");
}

template <int R>
int backward(const float* w, const float* k, const float* g, float* gw, float* gk, float* work, int most, int B, int C, int T, cudaStream_t st) {
    const cudaError_t e = allow_smem<timex_fft_backward_kernel<R>>(Plan<R>::kSmem);
    RWKV_REQUIRE(e == cudaSuccess, RWKVB200_ECUDA, "timex_backward: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    const int s = splits(B, C, Plan<R>::G, work != nullptr ? most : 1);
    timex_fft_backward_kernel<R><<<dim3(C, s), Plan<R>::kThreads, Plan<R>::kSmem, st>>>(w, k, g, s > 1 ? work : gw, gk, B, C, T);
    if (int rc = check_launch("timex_backward(transforms)")) return rc;
    return s > 1 ? sum_rows(RWKVB200_F32, s, C * T, work, gw, st) : RWKVB200_OK;
}

}  // namespace

// Up to 256 tokens the direct form is the more precise one: its error against fp64 is 1.48e-8 sqrt(T) of the norm, the
// transforms' is 1.9e-7 (256 points) to 2.4e-7 (2048) and falls below it between 256 and 257 tokens, where the transforms
// get longer (T = 256: 2.35e-7 direct, 2.43e-7 with 512 points; T = 257: 2.36e-7 direct, 2.14e-7 with 1024).  Above 1024 the
// engine has no transform long enough.
bool timex_fft_applies(int T) { return T > 256 && T <= 1024; }

// The shortest transform that holds T tokens and as many zeros.  (768 points, R = 3, for up to 384 tokens were no faster than 1024:
// B32 C768 T384 172 against 170 us.)
int timex_fft_forward(const float* w, const float* k, float* x, float eps, int B, int C, int T, cudaStream_t st) {
    return T <= 512 ? forward<4>(w, k, x, eps, B, C, T, st)
           : T <= 768 ? forward<6>(w, k, x, eps, B, C, T, st) : forward<8>(w, k, x, eps, B, C, T, st);
}
int timex_fft_backward(const float* w, const float* k, const float* g, float* gw, float* gk, float* work, int B, int C, int T, cudaStream_t st) {
    return T <= 512 ? backward<4>(w, k, g, gw, gk, work, kTimexSplits, B, C, T, st)
           : T <= 768 ? backward<6>(w, k, g, gw, gk, work, kTimexSplits, B, C, T, st) : backward<8>(w, k, g, gw, gk, work, kTimexSplits, B, C, T, st);
}

}  // namespace rwkvb200
