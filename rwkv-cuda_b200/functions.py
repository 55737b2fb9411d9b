"""torch.autograd.Function mirrors of the reference harnesses' operators: same class names, same arguments of `apply`,
same results.  Module-level globals of the reference (HEAD_SIZE, B, T, C ...) are taken from the tensors.

Where `apply` is given here, the whole call is native code with an autograd node of its own (csrc_py/native.cpp).  That node
answers None for calls that only torch.autograd.Function can take or refuse (jit tracing, forward-mode derivatives, functorch);
those, and subclasses, go through `forward` and `backward`, which run the same kernels.
"""
import torch

from . import ops
from ._lib import native


def _keep(ctx, made):
    """The outputs of a native forward; the rest of what it made is kept for `_gradients`."""
    out, kept, ctx.n_inputs, ctx.dims = made
    ctx.save_for_backward(*kept)
    return out


def _gradients(ctx, backward, *grads):
    return backward(ctx.saved_tensors, ctx.n_inputs, ctx.dims, grads)


class WKV(torch.autograd.Function):
    """RWKV-4 (wkv/run.py:89-117): w is time_decay; the harness's w -> -exp(w) before and its sums of the per-batch gw, gu
    after are done by the kernels."""

    @classmethod
    def apply(cls, B, T, C, w, u, k, v):
        out = native().wkv4(B, T, C, w, u, k, v) if cls is WKV else None
        return out if out is not None else super().apply(B, T, C, w, u, k, v)

    @staticmethod
    def forward(ctx, B, T, C, w, u, k, v):
        return _keep(ctx, native().wkv4_forward(B, T, C, w, u, k, v))

    @staticmethod
    def backward(ctx, gy):
        return None, None, None, *_gradients(ctx, native().wkv4_backward, gy)


class TimeX(torch.autograd.Function):
    """depthwise_conv1d (depthwise_conv1d/run.py:76-102); gw is reduced over the batch inside the kernels."""

    @classmethod
    def apply(cls, w, k, B, C, T, eps):
        out = native().timex(w, k, B, C, T, eps) if cls is TimeX else None
        return out if out is not None else super().apply(w, k, B, C, T, eps)

    @staticmethod
    def forward(ctx, w, k, B, C, T, eps):
        return _keep(ctx, native().timex_forward(w, k, B, C, T, eps))

    @staticmethod
    def backward(ctx, gwk):
        return *_gradients(ctx, native().timex_backward, gwk), None, None, None, None


class WKV_5(torch.autograd.Function):
    """RWKV-5, bf16 or fp32 (wkv5_bf16/run.py:44-88, wkv5/run.py:469-504): w is the raw decay input.  The harness sums bf16
    (B,C) partials of gw, gu in bf16 (wkv5_bf16/run.py:83-87); here they are summed in fp32 and rounded once."""

    @classmethod
    def apply(cls, B, T, C, H, r, k, v, w, u):
        out = native().wkv5(B, T, C, H, r, k, v, w, u) if cls is WKV_5 else None
        return out if out is not None else super().apply(B, T, C, H, r, k, v, w, u)

    @staticmethod
    def forward(ctx, B, T, C, H, r, k, v, w, u):
        return _keep(ctx, native().wkv5_forward(B, T, C, H, r, k, v, w, u))

    @staticmethod
    def backward(ctx, gy):
        return None, None, None, None, *_gradients(ctx, native().wkv5_backward, gy)


class WKV_5A(torch.autograd.Function):
    """RWKV-5a (wkv5a/run.py:100-154); r,k,v are (B,T,C), w1,u1,w2,u2 are (H,N)."""

    @staticmethod
    def forward(ctx, r, k, v, w1, u1, w2, u2):
        with torch.no_grad():
            B, T, C = r.shape
            H = w1.shape[0]
            ctx.dims = (B, T, C, H)
            r, k, v, w1, u1, w2, u2 = (x.contiguous() for x in (r, k, v, w1, u1, w2, u2))
            ew1 = (-torch.exp(w1.float())).contiguous()
            eew1 = torch.exp(ew1).contiguous()
            ew2 = (-torch.exp(w2.float())).contiguous()
            eew2 = torch.exp(ew2).contiguous()
            ctx.save_for_backward(r, k, v, eew1, ew1, u1, eew2, ew2, u2)
            y = torch.empty((B, T, C), device=r.device, dtype=r.dtype)
            ops.wkv5a_forward(B, T, C, H, r, k, v, eew1, u1, eew2, u2, y)
            return y

    @staticmethod
    def backward(ctx, gy):
        with torch.no_grad():
            B, T, C, H = ctx.dims
            r, k, v, eew1, ew1, u1, eew2, ew2, u2 = ctx.saved_tensors
            gr, gk, gv = (torch.empty((B, T, C), device=gy.device, dtype=r.dtype) for _ in range(3))
            gw1, gu1, gw2, gu2 = (torch.empty((B, C), device=gy.device, dtype=r.dtype) for _ in range(4))
            ops.wkv5a_backward(B, T, C, H, r, k, v, eew1, ew1, u1, eew2, ew2, u2, gy.contiguous(), gr, gk, gv, gw1,
                               gu1, gw2, gu2)
            return (gr, gk, gv, *(torch.sum(g, 0).view(H, C // H) for g in (gw1, gu1, gw2, gu2)))


class WKV_6(torch.autograd.Function):
    """RWKV-6 (wkv6/run.py:128-170).  The harness hands its kernel ew = -exp(w) in fp32; here the kernels take w itself
    (in the activation dtype) and keep the chunk-start states for the backward, as in WKV_6STATE_EX without a state.
    Only a w of another dtype than the activations goes the harness's way."""

    @classmethod
    def apply(cls, B, T, C, H, r, k, v, w, u):
        out = native().wkv6(B, T, C, H, r, k, v, w, u) if cls is WKV_6 and w.dtype == r.dtype else None
        return out if out is not None else super().apply(B, T, C, H, r, k, v, w, u)

    @staticmethod
    def forward(ctx, B, T, C, H, r, k, v, w, u):
        ctx.raw = w.dtype == r.dtype
        if ctx.raw:
            return _keep(ctx, native().wkv6_forward(B, T, C, H, r, k, v, w, u))
        with torch.no_grad():
            ctx.B, ctx.T, ctx.C, ctx.H = B, T, C, H
            r, k, v, w, u = (x.contiguous() for x in (r, k, v, w, u))
            ew = (-torch.exp(w.float())).contiguous()
            ctx.save_for_backward(r, k, v, ew, u)
            y = torch.empty((B, T, C), device=r.device, dtype=r.dtype)
            ops.wkv6_forward(B, T, C, H, r, k, v, ew, u, y)
            return y

    @staticmethod
    def backward(ctx, gy):
        if ctx.raw:
            return None, None, None, None, *_gradients(ctx, native().wkv6_backward, gy)
        with torch.no_grad():
            B, T, C, H = ctx.B, ctx.T, ctx.C, ctx.H
            r, k, v, ew, u = ctx.saved_tensors
            gr, gk, gv, gw = (torch.empty((B, T, C), device=gy.device, dtype=r.dtype) for _ in range(4))
            gu = torch.empty((B, C), device=gy.device, dtype=r.dtype)
            ops.wkv6_backward(B, T, C, H, r, k, v, ew, u, gy.contiguous(), gr, gk, gv, gw, gu)
            return (None, None, None, None, gr, gk, gv, gw, torch.sum(gu, 0).view(H, C // H))


class WKV_6STATE(torch.autograd.Function):
    """RWKV-6 with initial state (wkv6_state/run.py:80-124): everything in the activation dtype."""

    @staticmethod
    def forward(ctx, B, T, C, H, r, k, v, w, u, s):
        with torch.no_grad():
            ctx.B, ctx.T, ctx.C, ctx.H = B, T, C, H
            r, k, v, w, u, s = (x.contiguous() for x in (r, k, v, w, u, s))
            ctx.save_for_backward(r, k, v, w, u, s)
            y = torch.empty((B, T, C), device=r.device, dtype=r.dtype)
            ops.wkv6state_forward(B, T, C, H, r, k, v, w, u, s, y)
            return y

    @staticmethod
    def backward(ctx, gy):
        with torch.no_grad():
            B, T, C, H = ctx.B, ctx.T, ctx.C, ctx.H
            r, k, v, w, u, s = ctx.saved_tensors
            gr, gk, gv, gw = (torch.empty((B, T, C), device=gy.device, dtype=r.dtype) for _ in range(4))
            gu = torch.empty((B, C), device=gy.device, dtype=r.dtype)
            gs = torch.empty((B, H, C // H, C // H), device=gy.device, dtype=r.dtype)
            ops.wkv6state_backward(B, T, C, H, r, k, v, w, u, s, gy.contiguous(), gr, gk, gv, gw, gu, gs)
            return (None, None, None, None, gr, gk, gv, gw, torch.sum(gu, 0).view(H, C // H), gs)


class WKV_6STATE_EX(torch.autograd.Function):
    """RWKV-6 with fp32 state in and out (state passing), (r, k, v, w, u, s0) -> (y, sT); no counterpart class in the reference."""

    @classmethod
    def apply(cls, r, k, v, w, u, s0):
        out = native().wkv6_state(r, k, v, w, u, s0) if cls is WKV_6STATE_EX else None
        return out if out is not None else super().apply(r, k, v, w, u, s0)

    @staticmethod
    def forward(ctx, r, k, v, w, u, s0):
        return _keep(ctx, native().wkv6_state_forward(r, k, v, w, u, s0))

    @staticmethod
    def backward(ctx, gy, dsT):
        return tuple(_gradients(ctx, native().wkv6_state_backward, gy, dsT))


class RWKV7_CLAMPW_CUDA_OP(torch.autograd.Function):
    """rwkv7_fast_fused/rwkv7_cuda_benchmark.py:76-96; inputs (B,T,H,N)."""

    @classmethod
    def apply(cls, r, w, k, v, a, b):
        out = native().wkv7(r, w, k, v, a, b) if cls is RWKV7_CLAMPW_CUDA_OP else None
        return out if out is not None else super().apply(r, w, k, v, a, b)

    @staticmethod
    def forward(ctx, r, w, k, v, a, b):
        return _keep(ctx, native().wkv7_forward(r, w, k, v, a, b))

    @staticmethod
    def backward(ctx, dy):
        return tuple(_gradients(ctx, native().wkv7_backward, dy))


class RWKV7_STATE_CLAMPW_CUDA_OP(torch.autograd.Function):
    """rwkv7_fast_fused/rwkv7_cuda_benchmark_state.py:75-99."""

    @classmethod
    def apply(cls, s0, r, w, k, v, a, b):
        out = native().wkv7_state(s0, r, w, k, v, a, b) if cls is RWKV7_STATE_CLAMPW_CUDA_OP else None
        return out if out is not None else super().apply(s0, r, w, k, v, a, b)

    @staticmethod
    def forward(ctx, s0, r, w, k, v, a, b):
        return _keep(ctx, native().wkv7_state_forward(s0, r, w, k, v, a, b))

    @staticmethod
    def backward(ctx, dy):
        *grads, ds0 = _gradients(ctx, native().wkv7_state_backward, dy)
        return ds0, *grads


class RWKV7_STATE_PASSING_CLAMPW_CUDA_OP(torch.autograd.Function):
    """rwkv7_fast_fused/rwkv7_cuda_benchmark_state_passing.py:75-99: returns (y, sT)."""

    @classmethod
    def apply(cls, s0, r, w, k, v, a, b):
        out = native().wkv7_statepassing(s0, r, w, k, v, a, b) if cls is RWKV7_STATE_PASSING_CLAMPW_CUDA_OP else None
        return out if out is not None else super().apply(s0, r, w, k, v, a, b)

    @staticmethod
    def forward(ctx, s0, r, w, k, v, a, b):
        return _keep(ctx, native().wkv7_statepassing_forward(s0, r, w, k, v, a, b))

    @staticmethod
    def backward(ctx, dy, dsT):
        *grads, ds0 = _gradients(ctx, native().wkv7_statepassing_backward, dy, dsT)
        return ds0, *grads


def _heads(x, head_size):
    B, T, HC = x.shape
    return x.view(B, T, HC // head_size, head_size)


def RWKV7_CLAMPW_CUDA(r, w, k, v, a, b, head_size=64):
    B, T, HC = r.shape
    return RWKV7_CLAMPW_CUDA_OP.apply(*(_heads(i, head_size) for i in (r, w, k, v, a, b))).view(B, T, HC)


def RWKV7_STATE_CLAMPW_CUDA(s0, r, w, k, v, a, b):
    B, T, HC = r.shape
    return RWKV7_STATE_CLAMPW_CUDA_OP.apply(s0, *(_heads(i, s0.shape[-1]) for i in (r, w, k, v, a, b))).view(B, T, HC)


def RWKV7_STATE_PASSING_CLAMPW_CUDA(s0, r, w, k, v, a, b):
    return RWKV7_STATE_PASSING_CLAMPW_CUDA_OP.apply(s0, *(_heads(i, s0.shape[-1]) for i in (r, w, k, v, a, b)))
