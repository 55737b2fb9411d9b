// The host side of the training classes (functions.py) and of RWKV-7 inference (ops.wkv7_state_update) in native code.
//
// A small problem keeps the GPU busy for 5 to 50 us, and the same work in Python (the checks of eight tensors, the stream,
// the ctypes call, an autograd.Function written in Python and its re-entry from the autograd thread) took 15 us for a
// decoding step and about 100 us for a training step.  Here a call checks its tensors, allocates its outputs and enters the
// C ABI of librwkvb200.so without coming back to the interpreter.
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/extension.h>

#include "../../include/rwkvb200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
namespace py = pybind11;

PyObject* g_error_class = PyExc_RuntimeError;   // rwkv_cuda_b200.RwkvB200Error

// Raises `cls(msg)` in Python: from a call that Python made, or from a backward on an autograd thread.
[[noreturn]] void raise(PyObject* cls, const std::string& msg, bool on_autograd_thread) {
    py::gil_scoped_acquire gil;
    PyErr_SetString(cls, msg.c_str());
    if (!on_autograd_thread) throw py::error_already_set();
    python_error e;
    e.persist();
    throw e;
}
void check_rc(int rc, const char* what, bool on_autograd_thread = false) {
    if (rc >= 0) return;
    raise(g_error_class, std::string(what) + ": " + rwkvb200_strerror(rc) + " (" + std::to_string(rc) + "): " + rwkvb200_last_error(), on_autograd_thread);
}
void assert_py(bool ok, const char* msg) {
    if (!ok) raise(PyExc_AssertionError, msg, false);
}

// the checks of ops.py, in the same words
void on_device(const Tensor& t, const char* name) {
    TORCH_CHECK(t.defined() && t.is_cuda(), name, ": tensor must be on a CUDA device (there is no CPU path)");
}
void* ptr(const Tensor& t, const char* name, at::ScalarType d) {
    on_device(t, name);
    TORCH_CHECK(t.is_contiguous(), name, ": tensor must be contiguous");
    TORCH_CHECK_TYPE(t.scalar_type() == d, name, ": expected ", d, ", got ", t.scalar_type());
    return t.data_ptr();
}
void* opt(const Tensor& t, const char* name, at::ScalarType d) { return t.defined() ? ptr(t, name, d) : nullptr; }
void numel(const Tensor& t, int64_t n, const char* name) {
    TORCH_CHECK(t.numel() == n, name, ": expected ", n, " elements, got ", t.sizes());
}
int dt(const Tensor& t, const char* name) {
    if (t.scalar_type() == at::kFloat) return RWKVB200_F32;
    TORCH_CHECK_TYPE(t.scalar_type() == at::kBFloat16, name, ": dtype ", t.scalar_type(), " not supported (float32 or bfloat16)");
    return RWKVB200_BF16;
}
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
Tensor empty(at::IntArrayRef sizes, at::ScalarType d, const Tensor& like) {
    return Tensor(at::detail::empty_cuda(sizes, d, like.device(), std::nullopt));
}
Tensor bytes(size_t n, const Tensor& like) { return empty({(int64_t)n}, at::kByte, like); }
Tensor same(const Tensor& like) { return empty(like.sizes(), like.scalar_type(), like); }
const float* f32(const void* p) { return static_cast<const float*>(p); }
float* f32(void* p) { return static_cast<float*>(p); }

}  // namespace

// ---- RWKV-7 inference ---------------------------------------------------------------------------------------
static void wkv7_state_update(const Tensor& state, const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a,
                              const Tensor& b, const Tensor& y) {
    on_device(r, "r");
    TORCH_CHECK_VALUE(r.dim() == 4, "r: expected (B,T,H,N), got ", r.sizes());
    const c10::cuda::CUDAGuard guard(r.device());
    const auto d = r.scalar_type();
    const int dtype = dt(r, "r");
    check_rc(rwkvb200_wkv7_state_update(dtype, r.size(0), r.size(1), r.size(2), r.size(3), f32(ptr(state, "state", at::kFloat)), ptr(r, "r", d),
                                        ptr(w, "w", d), ptr(k, "k", d), ptr(v, "v", d), ptr(a, "a", d), ptr(b, "b", d), ptr(y, "y", d), stream()),
             "rwkvb200_wkv7_state_update");
}

// ---- RWKV-4 -------------------------------------------------------------------------------------------------
struct Wkv4 : torch::autograd::Function<Wkv4> {
    static Tensor forward(AutogradContext* ctx, int64_t B, int64_t T, int64_t C, Tensor w, Tensor u, Tensor k, Tensor v) {
        on_device(k, "k");
        const c10::cuda::CUDAGuard guard(k.device());
        const auto f = at::kFloat;
        w = w.contiguous(); u = u.contiguous(); k = k.contiguous(); v = v.contiguous();
        numel(w, C, "w"); numel(u, C, "u"); numel(k, B * T * C, "k"); numel(v, B * T * C, "v");
        Tensor y = empty({B, T, C}, f, k);
        Tensor saved = empty({(int64_t)rwkvb200_wkv4_saved_bytes(B, T, C)}, at::kByte, k);
        check_rc(rwkvb200_wkv4_train_forward(B, T, C, f32(ptr(w, "w", f)), f32(ptr(u, "u", f)), f32(ptr(k, "k", f)), f32(ptr(v, "v", f)),
                                             f32(y.data_ptr()), saved.data_ptr(), stream()),
                 "rwkvb200_wkv4_train_forward");
        ctx->save_for_backward({w, u, k, v, saved});
        ctx->saved_data["dims"] = std::vector<int64_t>{B, T, C};
        return y;
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        const auto s = ctx->get_saved_variables();
        const auto dims = ctx->saved_data["dims"].toIntVector();
        const int64_t B = dims[0], T = dims[1], C = dims[2];
        const c10::cuda::CUDAGuard guard(s[2].device());
        const auto f = at::kFloat;
        const Tensor gy = g[0].contiguous();
        numel(gy, B * T * C, "gy");
        Tensor gwu = empty({2, C}, f, gy), gk = empty({B, T, C}, f, gy), gv = empty({B, T, C}, f, gy);
        Tensor partial = B > 1 ? empty({B, 2, C}, f, gy) : Tensor();
        check_rc(rwkvb200_wkv4_train_backward(B, T, C, f32(s[0].data_ptr()), f32(s[1].data_ptr()), f32(s[2].data_ptr()), f32(s[3].data_ptr()),
                                              f32(ptr(gy, "gy", f)), s[4].data_ptr(), f32(gwu.data_ptr()),
                                              partial.defined() ? f32(partial.data_ptr()) : nullptr, f32(gk.data_ptr()), f32(gv.data_ptr()), stream()),
                 "rwkvb200_wkv4_train_backward", true);
        return {Tensor(), Tensor(), Tensor(), gwu.select(0, 0).view_as(s[0]), gwu.select(0, 1).view_as(s[1]), gk, gv};
    }
};

// ---- depthwise_conv1d -----------------------------------------------------------------------------------------
struct TimeX : torch::autograd::Function<TimeX> {
    static Tensor forward(AutogradContext* ctx, Tensor w, Tensor k, int64_t B, int64_t C, int64_t T, double eps) {
        on_device(k, "k");
        const c10::cuda::CUDAGuard guard(k.device());
        const auto f = at::kFloat;
        w = w.contiguous(); k = k.contiguous();
        numel(w, C * T, "w"); numel(k, B * C * T, "k");
        Tensor x = empty({B, C, T}, f, k);
        check_rc(rwkvb200_timex_forward(f32(ptr(w, "w", f)), f32(ptr(k, "k", f)), f32(x.data_ptr()), (float)eps, B, C, T, stream()), "rwkvb200_timex_forward");
        ctx->save_for_backward({w, k});
        ctx->saved_data["dims"] = std::vector<int64_t>{B, C, T};
        return x;
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        const auto s = ctx->get_saved_variables();
        const auto dims = ctx->saved_data["dims"].toIntVector();
        const int64_t B = dims[0], C = dims[1], T = dims[2];
        const c10::cuda::CUDAGuard guard(s[1].device());
        const auto f = at::kFloat;
        const Tensor gx = g[0].contiguous();
        numel(gx, B * C * T, "gwk");
        Tensor gw = empty({C, T}, f, gx), gk = empty({B, C, T}, f, gx);
        const size_t nbytes = rwkvb200_timex_work_bytes(B, C, T);
        Tensor work = nbytes ? bytes(nbytes, gx) : Tensor();
        check_rc(rwkvb200_timex_train_backward(f32(s[0].data_ptr()), f32(s[1].data_ptr()), f32(ptr(gx, "gwk", f)), f32(gw.data_ptr()),
                                               f32(gk.data_ptr()), nbytes ? f32(work.data_ptr()) : nullptr, B, C, T, stream()),
                 "rwkvb200_timex_train_backward", true);
        return {gw, gk, Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

// ---- RWKV-5 ---------------------------------------------------------------------------------------------------
struct Wkv5 : torch::autograd::Function<Wkv5> {
    static Tensor forward(AutogradContext* ctx, int64_t B, int64_t T, int64_t C, int64_t H, Tensor r, Tensor k, Tensor v, Tensor w, Tensor u) {
        for (const Tensor* x : {&k, &v, &w, &u}) assert_py(x->scalar_type() == r.scalar_type(), "r, k, v, w, u must have one dtype");
        on_device(r, "r");
        const c10::cuda::CUDAGuard guard(r.device());
        const auto d = r.scalar_type();
        const int dtype = dt(r, "r");
        r = r.contiguous(); k = k.contiguous(); v = v.contiguous(); w = w.contiguous(); u = u.contiguous();
        numel(r, B * T * C, "r"); numel(k, B * T * C, "k"); numel(v, B * T * C, "v"); numel(w, C, "w"); numel(u, C, "u");
        Tensor y = empty({B, T, C}, d, r), saved = bytes(rwkvb200_wkv5_train_saved_bytes(B, T, C, H), r);
        const int path = rwkvb200_wkv5_train_forward(dtype, B, T, C, H, ptr(r, "r", d), ptr(k, "k", d), ptr(v, "v", d), ptr(w, "w", d),
                                                     ptr(u, "u", d), y.data_ptr(), saved.data_ptr(), stream());
        check_rc(path, "rwkvb200_wkv5_train_forward");
        ctx->save_for_backward({r, k, v, w, u, saved});
        ctx->saved_data["dims"] = std::vector<int64_t>{B, T, C, H, path};
        return y;
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        const auto s = ctx->get_saved_variables();
        const auto dims = ctx->saved_data["dims"].toIntVector();
        const int64_t B = dims[0], T = dims[1], C = dims[2], H = dims[3], path = dims[4];
        const c10::cuda::CUDAGuard guard(s[0].device());
        const auto d = s[0].scalar_type();
        const Tensor gy = g[0].contiguous();
        numel(gy, B * T * C, "gy");
        Tensor gr = empty({B, T, C}, d, gy), gk = empty({B, T, C}, d, gy), gv = empty({B, T, C}, d, gy), gwu = empty({2, C}, d, gy);
        Tensor work = bytes(rwkvb200_wkv5_train_work_bytes(B, T, C, H, path), gy);
        check_rc(rwkvb200_wkv5_train_backward(dt(s[0], "r"), B, T, C, H, path, s[0].data_ptr(), s[1].data_ptr(), s[2].data_ptr(), s[3].data_ptr(),
                                              s[4].data_ptr(), ptr(gy, "gy", d), gr.data_ptr(), gk.data_ptr(), gv.data_ptr(), gwu.data_ptr(),
                                              s[5].data_ptr(), work.data_ptr(), stream()),
                 "rwkvb200_wkv5_train_backward", true);
        return {Tensor(), Tensor(), Tensor(), Tensor(), gr, gk, gv, gwu.select(0, 0).view_as(s[3]), gwu.select(0, 1).view_as(s[4])};
    }
};

// ---- RWKV-6, without a state (kState = false) or with an fp32 state in and out ----------------------------------------
template <bool kState>
struct Wkv6 : torch::autograd::Function<Wkv6<kState>> {
    static variable_list forward(AutogradContext* ctx, int64_t B, int64_t T, int64_t C, int64_t H, Tensor r, Tensor k, Tensor v, Tensor w,
                                 Tensor u, std::optional<Tensor> state) {
        on_device(r, "r");
        Tensor s0 = kState ? state->contiguous() : Tensor();
        const c10::cuda::CUDAGuard guard(r.device());
        const auto d = r.scalar_type(), f = at::kFloat;
        const int dtype = dt(r, "r");
        r = r.contiguous(); k = k.contiguous(); v = v.contiguous(); w = w.contiguous(); u = u.contiguous();
        numel(r, B * T * C, "r"); numel(k, B * T * C, "k"); numel(v, B * T * C, "v"); numel(w, B * T * C, "w"); numel(u, C, "u");
        if (kState) numel(s0, B * H * (C / H) * (C / H), "s0");
        Tensor y = empty({B, T, C}, d, r), sT = kState ? same(s0) : Tensor();
        Tensor saved = bytes(rwkvb200_wkv6_train_saved_bytes(dtype, B, T, C, H), r);
        const int path = rwkvb200_wkv6_train_forward(dtype, B, T, C, H, ptr(r, "r", d), ptr(k, "k", d), ptr(v, "v", d), ptr(w, "w", d), ptr(u, "u", d),
                                                     kState ? f32(ptr(s0, "s0", f)) : nullptr, y.data_ptr(), kState ? f32(sT.data_ptr()) : nullptr,
                                                     saved.data_ptr(), stream());
        check_rc(path, "rwkvb200_wkv6_train_forward");
        ctx->save_for_backward({r, k, v, w, u, saved, kState ? s0 : saved});
        ctx->saved_data["dims"] = std::vector<int64_t>{B, T, C, H, path};
        if (kState) return {y, sT};
        return {y};
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        const auto s = ctx->get_saved_variables();
        const auto dims = ctx->saved_data["dims"].toIntVector();
        const int64_t B = dims[0], T = dims[1], C = dims[2], H = dims[3], path = dims[4];
        const c10::cuda::CUDAGuard guard(s[0].device());
        const auto d = s[0].scalar_type(), f = at::kFloat;
        const Tensor gy = g[0].contiguous(), dsT = kState ? g[1].contiguous() : Tensor();
        numel(gy, B * T * C, "gy");
        Tensor gr = empty({B, T, C}, d, gy), gk = empty({B, T, C}, d, gy), gv = empty({B, T, C}, d, gy), gw = empty({B, T, C}, d, gy);
        Tensor gu = empty(s[4].sizes(), d, gy), ds0 = kState ? same(s[6]) : Tensor();
        Tensor work = bytes(rwkvb200_wkv6_train_work_bytes(B, T, C, path), gy);
        check_rc(rwkvb200_wkv6_train_backward(dt(s[0], "r"), B, T, C, H, path, s[0].data_ptr(), s[1].data_ptr(), s[2].data_ptr(), s[3].data_ptr(),
                                              s[4].data_ptr(), kState ? f32(s[6].data_ptr()) : nullptr, ptr(gy, "gy", d),
                                              kState ? f32(ptr(dsT, "dsT", f)) : nullptr, gr.data_ptr(), gk.data_ptr(), gv.data_ptr(), gw.data_ptr(),
                                              gu.data_ptr(), kState ? f32(ds0.data_ptr()) : nullptr, s[5].data_ptr(), work.data_ptr(), stream()),
                 "rwkvb200_wkv6_train_backward", true);
        return {Tensor(), Tensor(), Tensor(), Tensor(), gr, gk, gv, gw, gu, ds0};
    }
};

// ---- RWKV-7, the three operators: state in (s0) and out (sT) or not ---------------------------------------------
constexpr int64_t kChunkLen = 16;

template <bool kS0, bool kST>
struct Wkv7 : torch::autograd::Function<Wkv7<kS0, kST>> {
    static variable_list forward(AutogradContext* ctx, std::optional<Tensor> state, Tensor r, Tensor w, Tensor k, Tensor v, Tensor a, Tensor b) {
        const Tensor s0 = kS0 ? *state : Tensor();
        assert_py(r.dim() == 4 && r.size(1) % kChunkLen == 0, "T must be a multiple of 16");
        for (const Tensor* x : {&w, &k, &v, &a, &b}) assert_py(x->scalar_type() == r.scalar_type(), "r, w, k, v, a, b must have one dtype");
        for (const Tensor* x : {&r, &w, &k, &v, &a, &b}) assert_py(x->is_contiguous(), "r, w, k, v, a, b must be contiguous");
        if (kS0) assert_py(s0.scalar_type() == at::kFloat && s0.is_contiguous(), "s0 must be contiguous float32");
        on_device(r, "r");
        const c10::cuda::CUDAGuard guard(r.device());
        const auto d = r.scalar_type(), f = at::kFloat;
        const int dtype = dt(r, "r");
        const int64_t B = r.size(0), T = r.size(1), H = r.size(2), N = r.size(3);
        Tensor y = same(v), sT = kST ? same(s0) : Tensor();
        Tensor s = empty({B, H, T / kChunkLen, N, N}, f, r), sa = empty({B, T, H, N}, f, r);
        check_rc(rwkvb200_wkv7_forward(dtype, B, T, H, N, kChunkLen, kS0 ? f32(ptr(s0, "s0", f)) : nullptr, ptr(r, "r", d), ptr(w, "w", d),
                                       ptr(k, "k", d), ptr(v, "v", d), ptr(a, "a", d), ptr(b, "b", d), y.data_ptr(),
                                       kST ? f32(sT.data_ptr()) : nullptr, f32(s.data_ptr()), f32(sa.data_ptr()), stream()),
                 "rwkvb200_wkv7_forward");
        ctx->save_for_backward({r, w, k, v, a, b, s, sa});
        if (kST) return {y.view({B, T, H * N}), sT};
        return {y};
    }
    static variable_list backward(AutogradContext* ctx, variable_list g) {
        const auto x = ctx->get_saved_variables();
        const c10::cuda::CUDAGuard guard(x[0].device());
        const auto d = x[0].scalar_type(), f = at::kFloat;
        const int64_t B = x[0].size(0), T = x[0].size(1), H = x[0].size(2), N = x[0].size(3);
        const Tensor dy = g[0].contiguous(), dsT = kST ? g[1].contiguous() : Tensor();
        if (kST && dsT.scalar_type() != f) raise(PyExc_AssertionError, "dsT must be float32", true);
        Tensor ds0 = kS0 ? empty({B, H, N, N}, f, dy) : Tensor();
        variable_list out{ds0};
        for (int i = 0; i < 6; ++i) out.push_back(same(x[i]));
        check_rc(rwkvb200_wkv7_backward(dt(x[0], "r"), B, T, H, N, kChunkLen, x[0].data_ptr(), x[1].data_ptr(), x[2].data_ptr(), x[3].data_ptr(),
                                        x[4].data_ptr(), x[5].data_ptr(), ptr(dy, "dy", d), kST ? f32(ptr(dsT, "dsT", f)) : nullptr,
                                        f32(x[6].data_ptr()), f32(x[7].data_ptr()), kS0 ? f32(ds0.data_ptr()) : nullptr, out[1].data_ptr(),
                                        out[2].data_ptr(), out[3].data_ptr(), out[4].data_ptr(), out[5].data_ptr(), out[6].data_ptr(), stream()),
                 "rwkvb200_wkv7_backward", true);
        return out;
    }
};

PYBIND11_MODULE(_native, m) {
    m.def("set_error_class", [](py::object cls) { g_error_class = cls.inc_ref().ptr(); });
    m.def("wkv7_state_update", &wkv7_state_update);
    m.def("wkv4", [](int64_t B, int64_t T, int64_t C, const Tensor& w, const Tensor& u, const Tensor& k, const Tensor& v) {
        return Wkv4::apply(B, T, C, w, u, k, v);
    });
    m.def("timex", [](const Tensor& w, const Tensor& k, int64_t B, int64_t C, int64_t T, double eps) { return TimeX::apply(w, k, B, C, T, eps); });
    m.def("wkv5", [](int64_t B, int64_t T, int64_t C, int64_t H, const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w, const Tensor& u) {
        return Wkv5::apply(B, T, C, H, r, k, v, w, u);
    });
    m.def("wkv6", [](int64_t B, int64_t T, int64_t C, int64_t H, const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w, const Tensor& u) {
        return Wkv6<false>::apply(B, T, C, H, r, k, v, w, u, std::optional<Tensor>())[0];
    });
    m.def("wkv6_state", [](const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w, const Tensor& u, const Tensor& s0) {
        TORCH_CHECK_VALUE(r.dim() == 3, "r: expected (B,T,C), got ", r.sizes());
        const auto out = Wkv6<true>::apply(r.size(0), r.size(1), r.size(2), u.size(0), r, k, v, w, u, std::optional<Tensor>(s0));
        return std::make_tuple(out[0], out[1]);
    });
    m.def("wkv7", [](const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a, const Tensor& b) {
        return Wkv7<false, false>::apply(std::optional<Tensor>(), r, w, k, v, a, b)[0];
    });
    m.def("wkv7_state", [](const Tensor& s0, const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a, const Tensor& b) {
        return Wkv7<true, false>::apply(std::optional<Tensor>(s0), r, w, k, v, a, b)[0];
    });
    m.def("wkv7_statepassing", [](const Tensor& s0, const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a, const Tensor& b) {
        const auto out = Wkv7<true, true>::apply(std::optional<Tensor>(s0), r, w, k, v, a, b);
        return std::make_tuple(out[0], out[1]);
    });
}
