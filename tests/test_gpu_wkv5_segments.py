"""GPU parity of the RWKV-5 training classes where they run split over time in fp32 arithmetic (fp32 activations, head sizes
other than 64), against the fp64 oracle: lengths around a 32-token segment, every head-size instance, a decay of nearly 0."""
import pytest
import torch

from oracle import wkv_oracle as O
from tests import helpers as Hh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,N,lo,hi", [(torch.float32, 64, -6, -1), (torch.float32, 17, -6, -1), (torch.float32, 128, -6, 1),
                                           (torch.float32, 64, 2, 4), (torch.bfloat16, 32, -6, -1)])
@pytest.mark.parametrize("B,T,H", [(2, 2, 1), (1, 32, 2), (3, 33, 2), (2, 97, 3), (1, 300, 1)])
def test_rwkv5_segments(dtype, N, lo, hi, B, T, H):
    import rwkv_cuda_b200 as R
    g = Hh.gen(T + N)
    C = H * N
    xs = [0.5 * Hh.randn(g, B, T, C) for _ in range(3)] + [Hh.rand(g, H, N, lo=lo, hi=hi), Hh.rand(g, H, N, lo=-1, hi=1)]
    gy = Hh.randn(g, B, T, C).to(dtype)
    x64 = [x.to(dtype).double().requires_grad_(True) for x in xs]
    want = O.wkv5(*x64, H)
    want = [want.detach()] + list(torch.autograd.grad(want, x64, gy.double()))
    xd = [x.to(dtype).cuda().requires_grad_(True) for x in xs]
    got = R.functions.WKV_5.apply(B, T, C, H, *xd)
    got = [got.detach()] + list(torch.autograd.grad(got, xd, gy.cuda()))
    for a, b, name in zip(got, want, ("y", "gr", "gk", "gv", "gw", "gu")):
        if b.abs().max() > 0:
            Hh.assert_close(a, b, Hh.tol_for(dtype), f"wkv5 {name}")


@pytest.mark.parametrize("dtype,T", [(torch.float32, 2), (torch.bfloat16, 2), (torch.bfloat16, 16)])
def test_rwkv5_many_short_sequences(dtype, T):
    """More (batch, head) units than a grid has rows; every batch row is the same sequence, so the first one's results are all
    there is to check, and the gradients of w and u are its own times the number of rows."""
    import rwkv_cuda_b200 as R
    g = Hh.gen(T)
    B, H, N = 1100, 64, 64
    C = H * N
    xs = [0.5 * Hh.randn(g, 1, T, C) for _ in range(3)] + [Hh.rand(g, H, N, lo=-6, hi=-1), Hh.rand(g, H, N, lo=-1, hi=1)]
    gy = Hh.randn(g, 1, T, C).to(dtype)
    x64 = [x.to(dtype).double().requires_grad_(True) for x in xs]
    want = O.wkv5(*x64, H)
    want = [want.detach()] + list(torch.autograd.grad(want, x64, gy.double()))
    xd = [(x.to(dtype).cuda().expand(B, T, C).contiguous() if i < 3 else x.to(dtype).cuda()).requires_grad_(True) for i, x in enumerate(xs)]
    got = R.functions.WKV_5.apply(B, T, C, H, *xd)
    got = [got.detach()] + list(torch.autograd.grad(got, xd, gy.cuda().expand(B, T, C).contiguous()))
    for i, (a, b, name) in enumerate(zip(got, want, ("y", "gr", "gk", "gv", "gw", "gu"))):
        if i < 4:
            assert torch.equal(a, a[:1].expand_as(a)), name
            Hh.assert_close(a[:1], b, Hh.tol_for(dtype), name)
        else:
            Hh.assert_close(a.float() / B, b, Hh.tol_for(dtype), name)
