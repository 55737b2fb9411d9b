"""GPU tests of what the training classes are to autograd: nodes that a program may walk twice, with any inputs and gradients
that autograd can hand them."""
import pytest
import torch

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
