"""GPU tests of what the training classes are to autograd: nodes that a program may walk twice, with any inputs and gradients
that autograd can hand them."""
import pytest
import torch
import torch.utils.checkpoint

from oracle import wkv_oracle as O
from tests import helpers as Hh

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("state", [False, True])
def test_wkv6_walked_twice_with_a_strong_decay(state):
    """Head 1 decays too fast for the chunked form and is redone by the general-shape kernel; the second walk over the kept graph
    gives the first one's gradients, which are the oracle's."""
    import rwkv_cuda_b200 as R
    g = Hh.gen(3)
    B, T, H, N = 2, 64, 3, 64
    C = H * N
    r, k, v = (0.5 * Hh.randn(g, B, T, C) for _ in range(3))
    w = Hh.randn(g, B, T, H, N) - 5.0
    w[:, :, 1] += 7.0
    u, s0 = Hh.rand(g, H, N, lo=-1, hi=1), 0.1 * Hh.randn(g, B, H, N, N)
    gy, dsT = Hh.randn(g, B, T, C), Hh.randn(g, B, H, N, N)
    xs = [x.to(BF) for x in (r, k, v, w.view(B, T, C), u)] + ([s0] if state else [])
    xd = [x.cuda().requires_grad_(True) for x in xs]
    x64 = [x.double().requires_grad_(True) for x in xs]
    if state:
        out = R.functions.WKV_6STATE_EX.apply(*xd)
        gd = [gy.to(BF).cuda(), dsT.cuda()]
        want = O.wkv6(*x64[:5], H, s0=x64[5], return_state=True)
        want = torch.autograd.grad(want, x64, [gy.to(BF).double(), dsT.double()])
    else:
        out = R.functions.WKV_6.apply(B, T, C, H, *xd)
        gd = [gy.to(BF).cuda()]
        want = torch.autograd.grad(O.wkv6(*x64, H), x64, gy.to(BF).double())
    first = torch.autograd.grad(out, xd, gd, retain_graph=True)
    second = torch.autograd.grad(out, xd, gd, retain_graph=True)
    for a, b, x, name in zip(first, second, want, ("gr", "gk", "gv", "gw", "gu", "ds0")):
        Hh.assert_close(a, x, Hh.TOL_BF16, name)
        assert torch.equal(a, b), name


def cases():
    """name -> (inputs, call), small, every class whose node is native"""
    import rwkv_cuda_b200 as R
    F = R.functions
    g = Hh.gen(11)
    B, T, H, N = 2, 64, 2, 64
    C = H * N
    rkv = [(0.5 * Hh.randn(g, B, T, C)).to(BF) for _ in range(3)]
    w5, w6, u = (Hh.randn(g, H, N) - 3).to(BF), (Hh.randn(g, B, T, C) - 5).to(BF), Hh.rand(g, H, N, lo=-1, hi=1).to(BF)
    i7 = Hh.v7_inputs(B, 128, H, N, seed=5)
    x7 = [i7[n].to(BF).view(B, 128, H, N) for n in ("r", "w", "k", "v", "a", "b")]
    s0 = 0.1 * Hh.randn(g, B, H, N, N)
    return {
        "wkv4": ([Hh.randn(g, 32), Hh.randn(g, 32), Hh.randn(g, 2, 24, 32), Hh.randn(g, 2, 24, 32)], lambda *x: F.WKV.apply(2, 24, 32, *x)),
        "timex": ([Hh.randn(g, 8, 300) / 17, Hh.randn(g, 2, 8, 300)], lambda *x: F.TimeX.apply(*x, 2, 8, 300, 0.1)),
        "wkv5": ([*rkv, w5, u], lambda *x: F.WKV_5.apply(B, T, C, H, *x)),
        "wkv5 fp32": ([x.float() for x in (*rkv, w5, u)], lambda *x: F.WKV_5.apply(B, T, C, H, *x)),
        "wkv6": ([*rkv, w6, u], lambda *x: F.WKV_6.apply(B, T, C, H, *x)),
        "wkv6 state": ([*rkv, w6, u, s0], F.WKV_6STATE_EX.apply),
        "wkv7": (x7, F.RWKV7_CLAMPW_CUDA_OP.apply),
        "wkv7 state": ([s0, *x7], F.RWKV7_STATE_CLAMPW_CUDA_OP.apply),
        "wkv7 state passing": ([s0, *x7], F.RWKV7_STATE_PASSING_CLAMPW_CUDA_OP.apply),
    }


NAMES = ["wkv4", "timex", "wkv5", "wkv5 fp32", "wkv6", "wkv6 state", "wkv7", "wkv7 state", "wkv7 state passing"]


def outputs(y):
    return list(y) if isinstance(y, tuple) else [y]


def cotangents(ys):
    return [torch.cos(torch.arange(y.numel(), device=y.device, dtype=torch.float32)).view(y.shape).to(y.dtype) for y in ys]


def gradients(call, xs):
    ys = outputs(call(*xs))
    return torch.autograd.grad(ys, xs, cotangents(ys))


@pytest.mark.parametrize("name,strided", [(n, s) for n in NAMES for s in (False, True)
                                          if not (s and n.startswith("wkv7"))])   # (RWKV-7 takes contiguous tensors only)
def test_saved_tensor_hooks_see_all_that_is_kept(name, strided):
    """What the hooks do not hold is not needed: while they hold everything, a forward leaves nothing on the device but its
    outputs; gradients from tensors that went to the host and came back are the same."""
    xs, call = cases()[name]
    xs = [(torch.stack([x, x], -1).cuda()[..., 0] if strided else x.cuda()).requires_grad_(True) for x in xs]
    want = gradients(call, xs)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (t.cpu(), t.stride()), lambda p: p[0].cuda()):
        ys = outputs(call(*xs))
    held = torch.cuda.memory_allocated() - before
    room = sum((y.untyped_storage().nbytes() + 511) // 512 * 512 for y in ys)
    assert held <= room, f"{held} bytes stay on the device, the outputs are {room}"
    for a, b in zip(torch.autograd.grad(ys, xs, cotangents(ys)), want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("name", NAMES)
def test_checkpointing(name):
    xs, call = cases()[name]
    xs = [x.cuda().requires_grad_(True) for x in xs]
    want = gradients(call, xs)
    got = gradients(lambda *x: torch.utils.checkpoint.checkpoint(call, *x, use_reentrant=False), xs)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("name", ["wkv7 state", "wkv7 state passing"])
def test_rwkv7_state_carried_in_place(name):
    """The initial state may be overwritten between forward and backward, as a program does that carries it in one buffer."""
    xs, call = cases()[name]
    xs = [x.cuda().requires_grad_(i > 0) for i, x in enumerate(xs)]
    want = gradients(lambda *x: call(xs[0], *x), xs[1:])
    ys = outputs(call(*xs))
    xs[0].copy_(ys[1].detach() if len(ys) > 1 else torch.zeros_like(xs[0]))
    for a, b in zip(torch.autograd.grad(ys, xs[1:], cotangents(ys)), want):
        assert torch.equal(a, b)
