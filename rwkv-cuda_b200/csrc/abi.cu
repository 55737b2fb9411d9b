// Error plumbing, library identity and the RWKV-7 entry points (argument checks + dispatch
// between the general-shape kernels and the N = 64 tensor-core path).
#include "common.cuh"
#include "wkv7_dispatch.cuh"
#include "wkv6_chunked.cuh"
#include <atomic>
#include <initializer_list>

namespace rwkvb200 {

static thread_local char g_err[512] = "";

void set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}

int check_launch(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("%s: kernel launch failed: %s", what, cudaGetErrorString(e));
        return RWKVB200_ECUDA;
    }
    return RWKVB200_OK;
}

}  // namespace rwkvb200

using namespace rwkvb200;

extern "C" const char* rwkvb200_strerror(int code) {
    switch (code) {
        case RWKVB200_OK: return "ok";
        case RWKVB200_EINVAL: return "invalid argument";
        case RWKVB200_ENULL: return "null pointer";
        case RWKVB200_EALIGN: return "misaligned pointer";
        case RWKVB200_EUNSUPPORTED: return "unsupported configuration";
        case RWKVB200_ECUDA: return "CUDA error";
        default: return "unknown error";
    }
}

extern "C" const char* rwkvb200_last_error(void) { return g_err; }
extern "C" int rwkvb200_version(void) { return 100; }
extern "C" int rwkvb200_built_for_sm(void) { return 100; }

// 0 = automatic (tensor-core kernels where the shape allows), 1 = general-shape kernels only,
// 2 = tensor-core kernels or an error.  Read once per call; forward and backward of one operator call
// must see the same value (the saved buffers differ between the two kernel families).
static std::atomic<int> g_wkv7_path{0};
static std::atomic<int> g_wkv7_test_expire{0};
static std::atomic<int> g_wkv7_bwd_form{0};   // 0 automatic, 1 one-group kernels, 2 staged forward / two-stage backward

int rwkvb200::sm_count() {
    constexpr int kMaxDevices = 64;
    static std::atomic<int> cache[kMaxDevices] = {};
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
    if ((n = cache[dev].load()) != 0) return n;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    cache[dev].store(n);
    return n;
}

extern "C" int rwkvb200_wkv7_select_form(int form) {
    RWKV_REQUIRE(form >= 0 && form <= 2, RWKVB200_EINVAL, "wkv7_select_form: form %d not in 0..2", form);
    g_wkv7_bwd_form.store(form);
    return RWKVB200_OK;
}

extern "C" int rwkvb200_wkv7_select_path(int path) {
    RWKV_REQUIRE(path >= 0 && path <= 2, RWKVB200_EINVAL, "wkv7_select_path: path %d not in 0..2", path);
    g_wkv7_path.store(path);
    return RWKVB200_OK;
}

static std::atomic<int> g_no_tensor_maps{0};
bool rwkvb200::tensor_maps_disabled() { return g_no_tensor_maps.load() != 0; }
extern "C" int rwkvb200_test_disable_tensor_maps(int on) {
    g_no_tensor_maps.store(on ? 1 : 0);
    return RWKVB200_OK;
}

extern "C" int rwkvb200_wkv7_test_expire_next_forward(void) {
    g_wkv7_test_expire.store(1);
    return RWKVB200_OK;
}

static bool aligned16(std::initializer_list<const void*> ps) {
    for (const void* p : ps)
        if (p != nullptr && (reinterpret_cast<uintptr_t>(p) & 15) != 0) return false;
    return true;
}

// Forward and backward must agree on the layout of the saved buffers, so the choice depends
// on (path, dtype, N, chunk_len) only; misaligned tensors on the tensor-core path are an error.
static int wkv7_use_tensor_path(const char* what, int dtype, int N, int chunk, bool* use) {
    const int path = g_wkv7_path.load();
    const bool shape_ok = dtype == RWKVB200_BF16 && N == 64 && chunk == 16;
    if (path == 2)
        RWKV_REQUIRE(shape_ok, RWKVB200_EUNSUPPORTED, "%s: tensor-core path needs bf16, N=64, chunk_len=16", what);
    *use = shape_ok && path != 1;
    return RWKVB200_OK;
}

static int wkv7_check(const char* what, int dtype, int B, int T, int H, int N, int chunk) {
    RWKV_REQUIRE(dtype == RWKVB200_F32 || dtype == RWKVB200_BF16, RWKVB200_EINVAL, "%s: unknown dtype %d", what, dtype);
    RWKV_REQUIRE(B > 0 && T > 0 && H > 0 && N > 0 && chunk > 0, RWKVB200_EINVAL,
                 "%s: B=%d T=%d H=%d N=%d chunk_len=%d must be positive", what, B, T, H, N, chunk);
    RWKV_REQUIRE(B <= 65535, RWKVB200_EINVAL, "%s: B=%d exceeds 65535", what, B);
    RWKV_REQUIRE(N <= RWKVB200_MAX_HEAD_SIZE, RWKVB200_EUNSUPPORTED, "%s: head size %d > %d", what, N,
                 RWKVB200_MAX_HEAD_SIZE);
    RWKV_REQUIRE(T % chunk == 0, RWKVB200_EINVAL, "%s: T=%d is not a multiple of chunk_len=%d", what, T, chunk);
    return RWKVB200_OK;
}

extern "C" int rwkvb200_device_status(void) {
    const int f = wkv7_l32_fwd_error(), g = wkv7_l32_bwd_error();
    if (f < 0 || g < 0) {
        set_error("device_status: reading the status words failed");
        return RWKVB200_ECUDA;
    }
    const int p = wkv7_l32_bwdp_error(0), q = wkv7_l32_fwdp_error(0), r6 = wkv6_l32_error(0), b6 = wkv6_l32_bwd_error(0);
    const int v7s = wkv7_scan_error(0);
    if (p < 0 || q < 0 || r6 < 0 || b6 < 0 || v7s < 0) {
        set_error("device_status: reading the status words failed");
        return RWKVB200_ECUDA;
    }
    if (f) return 10 + f;
    if (g) return 20 + g;
    if (p) return p;            // the two-stage backward records 30.. (front group) or 40.. (back group)
    if (q) return q + 20;       // the staged RWKV-7 forward 50.. / 55.. / 60..
    if (r6) return r6 + 40;     // the staged RWKV-6 / RWKV-5 forward 70.. / 75.. / 80..
    if (b6) return b6 + 90;     // the tcgen05 RWKV-6 / RWKV-5 backward 91..
    return v7s ? v7s + 100 : 0; // the RWKV-7 kernels with the chunks in parallel 101..
}

extern "C" int rwkvb200_device_status_clear(void) {
    RWKV_REQUIRE(wkv7_l32_clear_errors() == 0 && wkv7_l32_bwdp_error(1) == 0 && wkv7_l32_fwdp_error(1) == 0 && wkv6_l32_error(1) == 0 && wkv6_l32_bwd_error(1) == 0 && wkv7_scan_error(1) == 0, RWKVB200_ECUDA, "device_status_clear: writing the status words failed");
    return RWKVB200_OK;
}

extern "C" int rwkvb200_wkv7_forward(int dtype, int B, int T, int H, int N, int chunk_len, const float* s0,
                                     const void* r, const void* w, const void* k, const void* v, const void* a,
                                     const void* b, void* y, float* sT, float* s, float* sa, void* stream) {
    if (int e = wkv7_check("wkv7_forward", dtype, B, T, H, N, chunk_len)) return e;
    RWKV_NOTNULL(r); RWKV_NOTNULL(w); RWKV_NOTNULL(k); RWKV_NOTNULL(v); RWKV_NOTNULL(a); RWKV_NOTNULL(b);
    RWKV_NOTNULL(y);
    RWKV_REQUIRE((s == nullptr) == (sa == nullptr), RWKVB200_EINVAL,
                 "wkv7_forward: s and sa must be given together (or both NULL for inference)");
    bool tensor;
    if (int e = wkv7_use_tensor_path("wkv7_forward", dtype, N, chunk_len, &tensor)) return e;
    if (tensor) {
        RWKV_REQUIRE(aligned16({s0, r, w, k, v, a, b, y, sT, s, sa}), RWKVB200_EALIGN,
                     "wkv7_forward: the bf16 N=64 path needs 16-byte aligned tensors");
        const int form = g_wkv7_bwd_form.load(), expire = g_wkv7_test_expire.exchange(0);
        // the staged form (three warp groups on consecutive chunks, inputs by TMA) is the faster one at every size
        if (!expire && form != 1) {
            const int rc = wkv7_l32_forward_pipelined(B, T, H, s0, r, w, k, v, a, b, y, sT, s, as_stream(stream));
            if (rc != 1) return rc;   // 1: no tensor maps on this driver, use the one-group kernel
        }
        return wkv7_l32_forward(B, T, H, s0, r, w, k, v, a, b, y, sT, s, expire, as_stream(stream));
    }
    return wkv7_generic_forward(dtype, B, T, H, N, chunk_len, s0, r, w, k, v, a, b, y, sT, s, sa, as_stream(stream));
}

extern "C" int rwkvb200_wkv7_backward(int dtype, int B, int T, int H, int N, int chunk_len, const void* r,
                                      const void* w, const void* k, const void* v, const void* a, const void* b,
                                      const void* dy, const float* dsT, const float* s, const float* sa, float* ds0,
                                      void* dr, void* dw, void* dk, void* dv, void* da, void* db, void* stream) {
    if (int e = wkv7_check("wkv7_backward", dtype, B, T, H, N, chunk_len)) return e;
    RWKV_NOTNULL(r); RWKV_NOTNULL(w); RWKV_NOTNULL(k); RWKV_NOTNULL(v); RWKV_NOTNULL(a); RWKV_NOTNULL(b);
    RWKV_NOTNULL(dy); RWKV_NOTNULL(s); RWKV_NOTNULL(sa);
    RWKV_NOTNULL(dr); RWKV_NOTNULL(dw); RWKV_NOTNULL(dk); RWKV_NOTNULL(dv); RWKV_NOTNULL(da); RWKV_NOTNULL(db);
    bool tensor;
    if (int e = wkv7_use_tensor_path("wkv7_backward", dtype, N, chunk_len, &tensor)) return e;
    if (tensor) {
        RWKV_REQUIRE(aligned16({r, w, k, v, a, b, dy, dsT, s, sa, ds0, dr, dw, dk, dv, da, db}), RWKVB200_EALIGN,
                     "wkv7_backward: the bf16 N=64 path needs 16-byte aligned tensors");
        // Two independent one-group blocks per SM give the most throughput while every place has a unit (8.6 k cycles per chunk
        // and SM); units that have an SM to themselves take the two-stage form (one block per SM, two warp groups on consecutive
        // chunks: 8.8 k cycles per chunk against 13.3 k).  So after one or two whole rounds of the one what is left over goes to the other,
        // where that is at most a unit per SM.  Forward + backward, us, one-group blocks only / this: one round and 24 to 148 units T512 345 to
        // 360 / 340 to 351, T1024 659 to 679 / 637 to 653, T4096 (B8 H40) 2533 / 2388; T256 187 / 190.  Two rounds T512 545 / 548, T1024 1043 / 1039,
        // T2048 2043 / 2020.  After three rounds the SMs are apart by so much that blocks of the last one start beside others: T512 744 / 757,
        // T1024 1428 / 1439, T2048 2797 / 2800, B16 T4096 H64 5592 / 5577 (two runs differ by 0.2 %; other boxes by 3 %).
        const int form = g_wkv7_bwd_form.load(), units = B * H, sms = sm_count(), places = 2 * sms, rounds = places > 0 ? units / places : 0;
        const bool tail = rounds >= 1 && rounds <= 2 && T >= 512 * rounds && units % places <= sms;
        const int rest = form == 1 ? 0 : form == 2 || units <= sms ? units : tail ? units % places : 0;
        if (units > rest)
            if (int e = wkv7_l32_backward(B, T, H, 0, units - rest, r, w, k, v, a, b, dy, dsT, s, ds0, dr, dw, dk, dv, da, db, as_stream(stream))) return e;
        if (rest == 0) return RWKVB200_OK;
        return wkv7_l32_backward_pipelined(B, T, H, units - rest, rest, r, w, k, v, a, b, dy, dsT, s, ds0, dr, dw, dk, dv, da, db, as_stream(stream));
    }
    return wkv7_generic_backward(dtype, B, T, H, N, chunk_len, r, w, k, v, a, b, dy, dsT, s, sa, ds0, dr, dw, dk, dv,
                                 da, db, as_stream(stream));
}

// Inference-shaped entry: advance the recurrent state by T >= 1 tokens in place and return y; nothing is
// saved for a backward pass and T needs no alignment (T = 1 is one decoding step).
extern "C" int rwkvb200_wkv7_state_update(int dtype, int B, int T, int H, int N, float* state, const void* r,
                                          const void* w, const void* k, const void* v, const void* a, const void* b,
                                          void* y, void* stream) {
    if (int e = wkv7_check("wkv7_state_update", dtype, B, T, H, N, 1)) return e;
    RWKV_NOTNULL(state); RWKV_NOTNULL(r); RWKV_NOTNULL(w); RWKV_NOTNULL(k); RWKV_NOTNULL(v); RWKV_NOTNULL(a); RWKV_NOTNULL(b);
    RWKV_NOTNULL(y);
    // long aligned prompts in bf16 with head size 64 take the tensor-core forward, decoding steps, odd lengths and fp32
    // the fp32 kernels of wkv7_update.cu, other head sizes the general-shape kernel
    const bool tensor = g_wkv7_path.load() != 1 && dtype == RWKVB200_BF16 && N == 64 && T % 16 == 0 && T >= 64 &&
                        aligned16({state, r, w, k, v, a, b, y});
    if (tensor) {
        if (g_wkv7_bwd_form.load() != 1) {
            const int rc = wkv7_l32_forward_pipelined(B, T, H, state, r, w, k, v, a, b, y, state, nullptr, as_stream(stream));
            if (rc != 1) return rc;   // 1: no tensor maps on this driver, use the one-group kernel
        }
        return wkv7_l32_forward(B, T, H, state, r, w, k, v, a, b, y, state, nullptr, 0, as_stream(stream));
    }
    if (N == 64 && aligned16({state, r, w, k, v, a, b, y}))
        return wkv7_update64(dtype, B, T, H, state, r, w, k, v, a, b, y, sm_count(), as_stream(stream));
    return wkv7_generic_forward(dtype, B, T, H, N, T, state, r, w, k, v, a, b, y, state, nullptr, nullptr, as_stream(stream));
}

// ---- training flow ------------------------------------------------------------------------------------------------------
// Path 1: the chunks in parallel (wkv7_scan.cu), for tensor-core shapes with at most a unit per two SMs: beyond that the extra
// products cost more than the short chain saves (T 2048, forward + backward: 32 units 408 -> 226 us, 64 units 410 -> 345 us,
// 80 units 413 -> 399 us, 128 units 421 -> 586 us), and up to 64 tokens there is next to nothing to walk in parallel.
// Its forward answers EUNSUPPORTED, with nothing enqueued, where the driver makes no tensor maps: the call is then one of path 0.
// Path 0: rwkvb200_wkv7_forward / _backward, `saved` = s then sa.
extern "C" int rwkvb200_wkv7_train_path(int dtype, int B, int T, int H, int N) {
    const bool tensor = dtype == RWKVB200_BF16 && N == 64 && g_wkv7_path.load() != 1 && g_wkv7_bwd_form.load() == 0;
    return tensor && T > 64 && 2ll * B * H <= sm_count() ? 1 : 0;
}
extern "C" size_t rwkvb200_wkv7_train_saved_bytes(int B, int T, int H, int N, int path) {
    if (B <= 0 || T <= 0 || H <= 0 || N <= 0) return 0;
    if (path == 1) return wkv7_scan_saved_bytes(B, T, H);
    return ((size_t)B * H * (T / 16) * N * N + (size_t)B * T * H * N) * sizeof(float);
}
extern "C" size_t rwkvb200_wkv7_train_work_bytes(int B, int T, int H, int path, int backward) {
    return path == 1 && B > 0 && T > 0 && H > 0 ? wkv7_scan_work_bytes(B, T, H, backward != 0) : 0;
}
extern "C" int rwkvb200_wkv7_train_forward(int dtype, int B, int T, int H, int N, int path, const float* s0, const void* r, const void* w,
                                           const void* k, const void* v, const void* a, const void* b, void* y, float* sT, void* saved,
                                           void* work, void* stream) {
    if (int e = wkv7_check("wkv7_train_forward", dtype, B, T, H, N, 16)) return e;
    RWKV_NOTNULL(saved);
    if (path == 0) {
        float* s = static_cast<float*>(saved);
        return rwkvb200_wkv7_forward(dtype, B, T, H, N, 16, s0, r, w, k, v, a, b, y, sT, s, s + (size_t)B * H * (T / 16) * N * N, stream);
    }
    RWKV_NOTNULL(r); RWKV_NOTNULL(w); RWKV_NOTNULL(k); RWKV_NOTNULL(v); RWKV_NOTNULL(a); RWKV_NOTNULL(b); RWKV_NOTNULL(y); RWKV_NOTNULL(work);
    RWKV_REQUIRE(dtype == RWKVB200_BF16 && N == 64, RWKVB200_EINVAL, "wkv7_train_forward: path 1 is bf16, head size 64");
    RWKV_REQUIRE(aligned16({s0, r, w, k, v, a, b, y, sT, saved, work}), RWKVB200_EALIGN, "wkv7_train_forward: the bf16 N=64 path needs 16-byte aligned tensors");
    const int rc = wkv7_scan_forward(B, T, H, s0, r, w, k, v, a, b, y, sT, saved, work, as_stream(stream));
    RWKV_REQUIRE(rc != 1, RWKVB200_EUNSUPPORTED, "wkv7_train_forward: tensor maps cannot be made here");
    return rc;
}
extern "C" int rwkvb200_wkv7_train_backward(int dtype, int B, int T, int H, int N, int path, const void* r, const void* w, const void* k,
                                            const void* v, const void* a, const void* b, const void* dy, const float* dsT, const void* saved,
                                            void* work, float* ds0, void* dr, void* dw, void* dk, void* dv, void* da, void* db, void* stream) {
    if (int e = wkv7_check("wkv7_train_backward", dtype, B, T, H, N, 16)) return e;
    RWKV_NOTNULL(saved);
    if (path == 0) {
        const float* s = static_cast<const float*>(saved);
        return rwkvb200_wkv7_backward(dtype, B, T, H, N, 16, r, w, k, v, a, b, dy, dsT, s, s + (size_t)B * H * (T / 16) * N * N, ds0, dr, dw, dk,
                                      dv, da, db, stream);
    }
    RWKV_NOTNULL(r); RWKV_NOTNULL(w); RWKV_NOTNULL(k); RWKV_NOTNULL(v); RWKV_NOTNULL(a); RWKV_NOTNULL(b); RWKV_NOTNULL(dy); RWKV_NOTNULL(work);
    RWKV_NOTNULL(dr); RWKV_NOTNULL(dw); RWKV_NOTNULL(dk); RWKV_NOTNULL(dv); RWKV_NOTNULL(da); RWKV_NOTNULL(db);
    RWKV_REQUIRE(dtype == RWKVB200_BF16 && N == 64, RWKVB200_EINVAL, "wkv7_train_backward: path 1 is bf16, head size 64");
    RWKV_REQUIRE(aligned16({r, w, k, v, a, b, dy, dsT, saved, work, ds0, dr, dw, dk, dv, da, db}), RWKVB200_EALIGN,
                 "wkv7_train_backward: the bf16 N=64 path needs 16-byte aligned tensors");
    return wkv7_scan_backward(B, T, H, r, w, k, v, a, b, dy, dsT, saved, work, ds0, dr, dw, dk, dv, da, db, as_stream(stream));
}
