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
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include "../../include/rwkvb200.h"

namespace {

using at::Tensor;
using torch::autograd::SavedVariable;
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
// a tensor of the shape of `like` on the storage of `whole`, from element `offset` on (without a trip through the dispatcher)
Tensor part(const Tensor& whole, int64_t offset, const Tensor& like) {
    Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(whole.storage()), whole.key_set(), whole.dtype());
    t.unsafeGetTensorImpl()->set_storage_offset(whole.storage_offset() + offset);
    t.unsafeGetTensorImpl()->set_sizes_contiguous(like.sizes());
    return t;
}

// Several outputs at once: one allocation when they are small (an allocation costs about 1 us, as much as a tenth of a small
// step), one each when keeping one of them alive would keep much memory alive.
struct Outputs {
    Tensor whole;
    int64_t at = 0;
    at::ScalarType d;
    Outputs(int64_t elems, int count, at::ScalarType type, const Tensor& like) : d(type) {
        if (elems * (int64_t)c10::elementSize(type) <= (1 << 20)) whole = empty({elems + 16 * count}, type, like);
    }
    Tensor next(at::IntArrayRef sizes, const Tensor& like) {
        if (!whole.defined()) return empty(sizes, d, like);
        Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(whole.storage()), whole.key_set(), whole.dtype());
        t.unsafeGetTensorImpl()->set_storage_offset(at);
        t.unsafeGetTensorImpl()->set_sizes_contiguous(sizes);
        at += (t.numel() + 15) / 16 * 16;   // 32-byte aligned
        return t;
    }
};

// ---- autograd -------------------------------------------------------------------------------------------------
// One node type for all operators (a node of its own instead of torch::autograd::Function, whose context, argument unpacking
// and dictionary cost as much as the launches): the inputs and the buffer that the forward made as saved variables (so that
// saved-tensor hooks, and with them checkpointing, see all that is kept), a few integers, and the operator's backward, which
// returns the gradients in the order of `inputs`.
struct Saved {
    std::array<Tensor, 8> in;       // contiguous inputs
    Tensor own;                     // buffer of the forward
    std::array<int64_t, 6> dims{};
};
// A saved tensor as it comes back, possibly out of a hook's hands.
Tensor unpacked(SavedVariable& x, at::ScalarType d, int64_t elements) {
    const Tensor t = x.unpack();
    TORCH_CHECK(t.defined() && t.is_cuda() && t.scalar_type() == d && t.numel() == elements,
                "saved tensor: expected ", elements, " elements of ", d, " on a CUDA device");
    return t.contiguous();
}
using BackwardFn = variable_list (*)(const Saved&, const variable_list& grads);

struct OpNode : torch::autograd::Node {
    BackwardFn fn = nullptr;
    const char* op = "";
    int n = 0;
    std::array<SavedVariable, 9> kept;   // the inputs, and behind them the forward's buffer
    std::array<at::ScalarType, 9> types;
    std::array<int64_t, 9> elements;
    std::array<int64_t, 6> dims{};
    bool released = false;

    std::string name() const override { return op; }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (auto& x : kept) x.reset_data();
        released = true;
    }
    variable_list apply(variable_list&& grads) override {
        Saved s;
        {
            std::lock_guard<std::mutex> lock(mutex_);
            TORCH_CHECK(!released, torch::autograd::ERR_BACKWARD_TWICE);
            for (int i = 0; i <= n; ++i)
                if (elements[i] != 0) (i < n ? s.in[i] : s.own) = unpacked(kept[i], types[i], elements[i]);
            s.dims = dims;
        }
        at::AutoDispatchBelowAutograd no_graph;
        for (size_t i = 0; i < grads.size(); ++i)
            grads[i] = grads[i].defined() ? grads[i].contiguous() : input_metadata(i).zeros_like();
        return fn(s, grads);
    }
};

// What a forward has made: the outputs, what is kept for the backward (s.in: contiguous forms of the inputs) and the backward.
struct Made {
    const char* op;
    BackwardFn backward;
    c10::SmallVector<Tensor, 2> outputs;
    c10::SmallVector<Tensor, 8> inputs;   // the differentiable ones, as given
    Saved s;
};

// Calls that are not for the node below: forward-mode derivatives, functorch's wrappers (grad, vmap, ...), tensors of classes
// with a dispatch of their own (and jit tracing).  torch.autograd.Function knows what to do with them.
bool ordinary(const Tensor& x) {
    constexpr c10::DispatchKeySet special({c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::Python});
    return !x.key_set().has_any(special) && !x._fw_grad(0).defined();
}
template <typename T>
bool ordinary(const T&) { return true; }   // (a number)

// Ties the outputs to a node that keeps what the forward has made.
void record(const Made& m) {
    const auto& inputs = m.inputs;
    const Saved& s = m.s;
    bool any = false;
    for (const Tensor& x : inputs) any |= x.requires_grad();
    if (!any || !at::GradMode::is_enabled()) return;
    auto node = std::shared_ptr<OpNode>(new OpNode(), torch::autograd::deleteNode);
    torch::autograd::edge_list edges;
    edges.reserve(inputs.size());
    for (const Tensor& x : inputs) edges.push_back(torch::autograd::impl::gradient_edge(x));
    node->set_next_edges(std::move(edges));
    node->fn = m.backward;
    node->op = m.op;
    node->n = inputs.size();
    for (int i = 0; i <= node->n; ++i) {   // (s.in[i]: the input, or the contiguous copy that had to be made of it)
        const Tensor& x = i < node->n ? s.in[i] : s.own;
        node->elements[i] = x.defined() ? x.numel() : 0;
        if (!x.defined()) continue;
        node->types[i] = x.scalar_type();
        node->kept[i] = SavedVariable(x, false);
    }
    node->dims = s.dims;
    for (const Tensor& y : m.outputs) torch::autograd::set_history(y, node);
}
Tensor dense(const Tensor& x) {   // contiguous form, outside of the graph
    if (x.is_contiguous()) return x;
    at::NoGradGuard guard;
    return x.contiguous();
}

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
static variable_list wkv4_backward(const Saved& s, const variable_list& g) {
    const auto [B, T, C, d3, d4, d5] = s.dims;
    const c10::cuda::CUDAGuard guard(s.in[2].device());
    const auto f = at::kFloat;
    const Tensor& gy = g[0];
    numel(gy, B * T * C, "gy");
    const int64_t n = B * T * C;
    Outputs o(2 * n + 2 * C + 2 * B * C, 4, f, gy);
    Tensor gk = o.next({B, T, C}, gy), gv = o.next({B, T, C}, gy), gwu = o.next({2, C}, gy);
    const Tensor partial = B > 1 ? o.next({B, 2, C}, gy) : Tensor();
    check_rc(rwkvb200_wkv4_train_backward(B, T, C, f32(s.in[0].data_ptr()), f32(s.in[1].data_ptr()), f32(s.in[2].data_ptr()),
                                          f32(s.in[3].data_ptr()), f32(ptr(gy, "gy", f)), s.own.data_ptr(), f32(gwu.data_ptr()),
                                          partial.defined() ? f32(partial.data_ptr()) : nullptr, f32(gk.data_ptr()), f32(gv.data_ptr()), stream()),
             "rwkvb200_wkv4_train_backward", true);
    return {part(gwu, 0, s.in[0]), part(gwu, C, s.in[1]), std::move(gk), std::move(gv)};
}
static Made wkv4(int64_t B, int64_t T, int64_t C, const Tensor& w, const Tensor& u, const Tensor& k, const Tensor& v) {
    on_device(k, "k");
    const c10::cuda::CUDAGuard guard(k.device());
    const auto f = at::kFloat;
    Saved s{{dense(w), dense(u), dense(k), dense(v)}, {}, {B, T, C}};
    numel(w, C, "w"); numel(u, C, "u"); numel(k, B * T * C, "k"); numel(v, B * T * C, "v");
    Tensor y = empty({B, T, C}, f, k);
    s.own = bytes(rwkvb200_wkv4_saved_bytes(B, T, C), k);
    check_rc(rwkvb200_wkv4_train_forward(B, T, C, f32(ptr(s.in[0], "w", f)), f32(ptr(s.in[1], "u", f)), f32(ptr(s.in[2], "k", f)),
                                         f32(ptr(s.in[3], "v", f)), f32(y.data_ptr()), s.own.data_ptr(), stream()),
             "rwkvb200_wkv4_train_forward");
    return {"WKVBackward", wkv4_backward, {y}, {w, u, k, v}, std::move(s)};
}

// ---- depthwise_conv1d -----------------------------------------------------------------------------------------
static variable_list timex_backward(const Saved& s, const variable_list& g) {
    const auto [B, C, T, d3, d4, d5] = s.dims;
    const c10::cuda::CUDAGuard guard(s.in[1].device());
    const auto f = at::kFloat;
    const Tensor& gx = g[0];
    numel(gx, B * C * T, "gwk");
    Outputs o(C * T + B * C * T, 2, f, gx);
    Tensor gw = o.next({C, T}, gx), gk = o.next({B, C, T}, gx);
    const size_t nbytes = rwkvb200_timex_work_bytes(B, C, T);
    const Tensor work = nbytes ? bytes(nbytes, gx) : Tensor();
    check_rc(rwkvb200_timex_train_backward(f32(s.in[0].data_ptr()), f32(s.in[1].data_ptr()), f32(ptr(gx, "gwk", f)), f32(gw.data_ptr()),
                                           f32(gk.data_ptr()), nbytes ? f32(work.data_ptr()) : nullptr, B, C, T, stream()),
             "rwkvb200_timex_train_backward", true);
    return {std::move(gw), std::move(gk)};
}
static Made timex(const Tensor& w, const Tensor& k, int64_t B, int64_t C, int64_t T, double eps) {
    on_device(k, "k");
    const c10::cuda::CUDAGuard guard(k.device());
    const auto f = at::kFloat;
    Saved s{{dense(w), dense(k)}, {}, {B, C, T}};
    numel(w, C * T, "w"); numel(k, B * C * T, "k");
    Tensor x = empty({B, C, T}, f, k);
    check_rc(rwkvb200_timex_forward(f32(ptr(s.in[0], "w", f)), f32(ptr(s.in[1], "k", f)), f32(x.data_ptr()), (float)eps, B, C, T, stream()),
             "rwkvb200_timex_forward");
    return {"TimeXBackward", timex_backward, {x}, {w, k}, std::move(s)};
}

// ---- RWKV-5 ---------------------------------------------------------------------------------------------------
static variable_list wkv5_backward(const Saved& s, const variable_list& g) {
    const auto [B, T, C, H, path, d5] = s.dims;
    const c10::cuda::CUDAGuard guard(s.in[0].device());
    const auto d = s.in[0].scalar_type();
    const Tensor& gy = g[0];
    numel(gy, B * T * C, "gy");
    Outputs o(3 * B * T * C + 2 * C, 4, d, gy);
    Tensor gr = o.next({B, T, C}, gy), gk = o.next({B, T, C}, gy), gv = o.next({B, T, C}, gy), gwu = o.next({2, C}, gy);
    const Tensor work = bytes(rwkvb200_wkv5_train_work_bytes(B, T, C, H, path), gy);
    check_rc(rwkvb200_wkv5_train_backward(dt(s.in[0], "r"), B, T, C, H, path, s.in[0].data_ptr(), s.in[1].data_ptr(), s.in[2].data_ptr(),
                                          s.in[3].data_ptr(), s.in[4].data_ptr(), ptr(gy, "gy", d), gr.data_ptr(), gk.data_ptr(), gv.data_ptr(),
                                          gwu.data_ptr(), s.own.data_ptr(), work.data_ptr(), stream()),
             "rwkvb200_wkv5_train_backward", true);
    return {std::move(gr), std::move(gk), std::move(gv), part(gwu, 0, s.in[3]), part(gwu, C, s.in[4])};
}
static Made wkv5(int64_t B, int64_t T, int64_t C, int64_t H, const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w, const Tensor& u) {
    for (const Tensor* x : {&k, &v, &w, &u}) assert_py(x->scalar_type() == r.scalar_type(), "r, k, v, w, u must have one dtype");
    on_device(r, "r");
    const c10::cuda::CUDAGuard guard(r.device());
    const auto d = r.scalar_type();
    const int dtype = dt(r, "r");
    Saved s{{dense(r), dense(k), dense(v), dense(w), dense(u)}, {}, {B, T, C, H}};
    numel(r, B * T * C, "r"); numel(k, B * T * C, "k"); numel(v, B * T * C, "v"); numel(w, C, "w"); numel(u, C, "u");
    Tensor y = empty({B, T, C}, d, r);
    s.own = bytes(rwkvb200_wkv5_train_saved_bytes(B, T, C, H), r);
    const int path = rwkvb200_wkv5_train_forward(dtype, B, T, C, H, ptr(s.in[0], "r", d), ptr(s.in[1], "k", d), ptr(s.in[2], "v", d),
                                                 ptr(s.in[3], "w", d), ptr(s.in[4], "u", d), y.data_ptr(), s.own.data_ptr(), stream());
    check_rc(path, "rwkvb200_wkv5_train_forward");
    s.dims[4] = path;
    return {"WKV_5Backward", wkv5_backward, {y}, {r, k, v, w, u}, std::move(s)};
}

// ---- RWKV-6, without a state or with an fp32 state in and out (s0, sT, dsT, ds0) ------------------------------------------
static variable_list wkv6_backward(const Saved& s, const variable_list& g) {
    const auto [B, T, C, H, path, state] = s.dims;
    const c10::cuda::CUDAGuard guard(s.in[0].device());
    const auto d = s.in[0].scalar_type(), f = at::kFloat;
    const Tensor& gy = g[0];
    numel(gy, B * T * C, "gy");
    Outputs o(4 * B * T * C + C, 5, d, gy);
    Tensor gr = o.next({B, T, C}, gy), gk = o.next({B, T, C}, gy), gv = o.next({B, T, C}, gy), gw = o.next({B, T, C}, gy);
    Tensor gu = o.next(s.in[4].sizes(), gy), ds0 = state ? same(s.in[5]) : Tensor();
    const Tensor work = bytes(rwkvb200_wkv6_train_work_bytes(B, T, C, path), gy);
    check_rc(rwkvb200_wkv6_train_backward(dt(s.in[0], "r"), B, T, C, H, path, s.in[0].data_ptr(), s.in[1].data_ptr(), s.in[2].data_ptr(),
                                          s.in[3].data_ptr(), s.in[4].data_ptr(), state ? f32(s.in[5].data_ptr()) : nullptr, ptr(gy, "gy", d),
                                          state ? f32(ptr(g[1], "dsT", f)) : nullptr, gr.data_ptr(), gk.data_ptr(), gv.data_ptr(), gw.data_ptr(),
                                          gu.data_ptr(), state ? f32(ds0.data_ptr()) : nullptr, s.own.data_ptr(), work.data_ptr(), stream()),
             "rwkvb200_wkv6_train_backward", true);
    variable_list out{std::move(gr), std::move(gk), std::move(gv), std::move(gw), std::move(gu)};
    if (state) out.push_back(std::move(ds0));
    return out;
}
static Made wkv6_forward(int64_t B, int64_t T, int64_t C, int64_t H, const Tensor& r, const Tensor& k, const Tensor& v,
                                               const Tensor& w, const Tensor& u, const Tensor* s0) {
    on_device(r, "r");
    const c10::cuda::CUDAGuard guard(r.device());
    const auto d = r.scalar_type(), f = at::kFloat;
    const int dtype = dt(r, "r");
    Saved s{{dense(r), dense(k), dense(v), dense(w), dense(u)}, {}, {B, T, C, H, 0, s0 != nullptr}};
    numel(r, B * T * C, "r"); numel(k, B * T * C, "k"); numel(v, B * T * C, "v"); numel(w, B * T * C, "w"); numel(u, C, "u");
    Tensor y = empty({B, T, C}, d, r), sT;
    if (s0) {
        numel(*s0, B * H * (C / H) * (C / H), "s0");
        s.in[5] = dense(*s0);
        sT = same(*s0);
    }
    s.own = bytes(rwkvb200_wkv6_train_saved_bytes(dtype, B, T, C, H), r);
    const int path = rwkvb200_wkv6_train_forward(dtype, B, T, C, H, ptr(s.in[0], "r", d), ptr(s.in[1], "k", d), ptr(s.in[2], "v", d),
                                                 ptr(s.in[3], "w", d), ptr(s.in[4], "u", d), s0 ? f32(ptr(s.in[5], "s0", f)) : nullptr,
                                                 y.data_ptr(), s0 ? f32(sT.data_ptr()) : nullptr, s.own.data_ptr(), stream());
    check_rc(path, "rwkvb200_wkv6_train_forward");
    s.dims[4] = path;
    if (s0) return {"WKV_6STATE_EXBackward", wkv6_backward, {y, sT}, {r, k, v, w, u, *s0}, std::move(s)};
    return {"WKV_6Backward", wkv6_backward, {y}, {r, k, v, w, u}, std::move(s)};
}

// ---- RWKV-7, the three operators: state in (s0) and out (sT) or not ---------------------------------------------
constexpr int64_t kChunkLen = 16;

static variable_list wkv7_backward(const Saved& s, const variable_list& g) {
    const auto [B, T, H, N, form, path] = s.dims;
    const bool s0 = form & 1, sT = form & 2;
    const c10::cuda::CUDAGuard guard(s.in[0].device());
    const auto d = s.in[0].scalar_type(), f = at::kFloat;
    if (sT && g[1].scalar_type() != f) raise(PyExc_AssertionError, "dsT must be float32", true);
    std::array<Tensor, 6> x;
    Outputs o(6 * B * T * H * N, 6, d, g[0]);
    for (auto& t : x) t = o.next({B, T, H, N}, g[0]);
    Tensor ds0 = s0 ? empty({B, H, N, N}, f, g[0]) : Tensor();
    const size_t nwork = rwkvb200_wkv7_train_work_bytes(B, T, H, path, 1);
    const Tensor work = nwork ? bytes(nwork, g[0]) : Tensor();
    check_rc(rwkvb200_wkv7_train_backward(dt(s.in[0], "r"), B, T, H, N, path, s.in[0].data_ptr(), s.in[1].data_ptr(), s.in[2].data_ptr(),
                                          s.in[3].data_ptr(), s.in[4].data_ptr(), s.in[5].data_ptr(), ptr(g[0], "dy", d),
                                          sT ? f32(ptr(g[1], "dsT", f)) : nullptr, s.own.data_ptr(), nwork ? work.data_ptr() : nullptr,
                                          s0 ? f32(ds0.data_ptr()) : nullptr, x[0].data_ptr(), x[1].data_ptr(), x[2].data_ptr(), x[3].data_ptr(),
                                          x[4].data_ptr(), x[5].data_ptr(), stream()),
             "rwkvb200_wkv7_train_backward", true);
    variable_list out{std::move(x[0]), std::move(x[1]), std::move(x[2]), std::move(x[3]), std::move(x[4]), std::move(x[5])};
    if (s0) out.push_back(std::move(ds0));
    return out;
}
static Made wkv7_forward(const Tensor* s0, const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v,
                                               const Tensor& a, const Tensor& b, bool passing) {
    assert_py(r.dim() == 4 && r.size(1) % kChunkLen == 0, "T must be a multiple of 16");
    for (const Tensor* x : {&w, &k, &v, &a, &b}) assert_py(x->scalar_type() == r.scalar_type(), "r, w, k, v, a, b must have one dtype");
    for (const Tensor* x : {&r, &w, &k, &v, &a, &b}) assert_py(x->is_contiguous(), "r, w, k, v, a, b must be contiguous");
    if (s0) assert_py(s0->scalar_type() == at::kFloat && s0->is_contiguous(), "s0 must be contiguous float32");
    on_device(r, "r");
    const c10::cuda::CUDAGuard guard(r.device());
    const auto d = r.scalar_type(), f = at::kFloat;
    const int dtype = dt(r, "r");
    const int64_t B = r.size(0), T = r.size(1), H = r.size(2), N = r.size(3);
    Tensor y = passing ? empty({B, T, H * N}, d, r) : same(v), sT = passing ? same(*s0) : Tensor();
    Saved s{{r, w, k, v, a, b}, {}, {B, T, H, N, (s0 ? 1 : 0) + (passing ? 2 : 0)}};
    auto run = [&](int path) {
        s.dims[5] = path;
        s.own = bytes(rwkvb200_wkv7_train_saved_bytes(B, T, H, N, path), r);
        const size_t nwork = rwkvb200_wkv7_train_work_bytes(B, T, H, path, 0);
        const Tensor work = nwork ? bytes(nwork, r) : Tensor();
        return rwkvb200_wkv7_train_forward(dtype, B, T, H, N, path, s0 ? f32(ptr(*s0, "s0", f)) : nullptr, ptr(r, "r", d), ptr(w, "w", d),
                                           ptr(k, "k", d), ptr(v, "v", d), ptr(a, "a", d), ptr(b, "b", d), y.data_ptr(),
                                           passing ? f32(sT.data_ptr()) : nullptr, s.own.data_ptr(), nwork ? work.data_ptr() : nullptr, stream());
    };
    const int path = rwkvb200_wkv7_train_path(dtype, B, T, H, N);
    int rc = run(path);
    if (rc == RWKVB200_EUNSUPPORTED && path != 0) rc = run(0);   // no tensor maps here: path 0 has kernels without
    check_rc(rc, "rwkvb200_wkv7_train_forward");
    // (the backward does not read s0: it is not kept, so that a program may carry its state in place)
    if (passing) return {"RWKV7_STATE_PASSING_CLAMPW_CUDA_OPBackward", wkv7_backward, {y, sT}, {r, w, k, v, a, b, *s0}, std::move(s)};
    if (s0) return {"RWKV7_STATE_CLAMPW_CUDA_OPBackward", wkv7_backward, {y}, {r, w, k, v, a, b, *s0}, std::move(s)};
    return {"RWKV7_CLAMPW_CUDA_OPBackward", wkv7_backward, {y}, {r, w, k, v, a, b}, std::move(s)};
}
static Made wkv6(int64_t B, int64_t T, int64_t C, int64_t H, const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w, const Tensor& u) {
    return wkv6_forward(B, T, C, H, r, k, v, w, u, nullptr);
}
static Made wkv6_state(const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w, const Tensor& u, const Tensor& s0) {
    TORCH_CHECK_VALUE(r.dim() == 3, "r: expected (B,T,C), got ", r.sizes());
    return wkv6_forward(r.size(0), r.size(1), r.size(2), u.size(0), r, k, v, w, u, &s0);
}
static Made wkv7(const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a, const Tensor& b) {
    return wkv7_forward(nullptr, r, w, k, v, a, b, false);
}
static Made wkv7_state(const Tensor& s0, const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a, const Tensor& b) {
    return wkv7_forward(&s0, r, w, k, v, a, b, false);
}
static Made wkv7_statepassing(const Tensor& s0, const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v, const Tensor& a, const Tensor& b) {
    return wkv7_forward(&s0, r, w, k, v, a, b, true);
}

// ---- bindings -----------------------------------------------------------------------------------------------
// A launch may wait for room in the GPU's queue: other Python threads run meanwhile.
template <typename F>
static auto unlocked(F f) {
    py::gil_scoped_release no_gil;
    return f();
}

// name: the outputs with their graph, or None for a call that is not for the native node.
// name_forward: the outputs, the tensors and integers that name_backward wants, and nothing recorded.
template <typename... A>
static void define(py::module_& m, const char* op_name, Made (*op)(A...), BackwardFn backward) {
    const std::string name = op_name;
    m.def(op_name, [op](A... args) -> py::object {
        bool plain = !torch::jit::tracer::isTracing();
        ((plain = plain && ordinary(args)), ...);
        if (!plain) return py::none();
        const Made r = unlocked([&] {
            Made made = op(args...);
            record(made);
            return made;
        });
        return r.outputs.size() == 1 ? py::cast(r.outputs[0]) : py::object(py::make_tuple(r.outputs[0], r.outputs[1]));
    });
    m.def((name + "_forward").c_str(), [op](A... args) {
        const Made r = unlocked([&] { return op(args...); });
        std::vector<Tensor> kept;
        for (size_t i = 0; i < r.s.in.size(); ++i)
            if (r.s.in[i].defined()) kept.push_back(r.s.in[i]);
        const size_t n = kept.size();
        if (r.s.own.defined()) kept.push_back(r.s.own);
        py::object y = r.outputs.size() == 1 ? py::cast(r.outputs[0]) : py::object(py::make_tuple(r.outputs[0], r.outputs[1]));
        return py::make_tuple(y, py::tuple(py::cast(kept)), n, r.s.dims);
    });
    m.def((name + "_backward").c_str(), [backward](const std::vector<Tensor>& kept, size_t n, const std::array<int64_t, 6>& dims, variable_list grads) {
        Saved s;
        s.dims = dims;
        for (size_t i = 0; i < kept.size(); ++i) (i < n ? s.in.at(i) : s.own) = kept[i].contiguous();
        return unlocked([&] {
            for (Tensor& g : grads) g = g.contiguous();
            return backward(s, grads);
        });
    });
}

PYBIND11_MODULE(_native, m) {
    m.def("set_error_class", [](py::object cls) { g_error_class = cls.inc_ref().ptr(); });
    m.def("wkv7_state_update", &wkv7_state_update, py::call_guard<py::gil_scoped_release>());
    define(m, "wkv4", &wkv4, wkv4_backward);
    define(m, "timex", &timex, timex_backward);
    define(m, "wkv5", &wkv5, wkv5_backward);
    define(m, "wkv6", &wkv6, wkv6_backward);
    define(m, "wkv6_state", &wkv6_state, wkv6_backward);
    define(m, "wkv7", &wkv7, wkv7_backward);
    define(m, "wkv7_state", &wkv7_state, wkv7_backward);
    define(m, "wkv7_statepassing", &wkv7_statepassing, wkv7_backward);
}
