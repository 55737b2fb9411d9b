"""GPU parity of depthwise_conv1d by transforms against the fp64 oracle: lengths on both sides of every transform length, odd
batches (a pair with one row) and batches that are split over blocks."""
import pytest
import torch

from oracle import wkv_oracle as O
from tests import helpers as Hh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [64, 65, 128, 129, 256, 257, 512, 513, 1024, 1025])
@pytest.mark.parametrize("B,C", [(1, 3), (3, 2), (33, 2)])
def test_conv1d_training_class(B, C, T):
    import rwkv_cuda_b200 as R
    g = Hh.gen(T + B)
    xs = [Hh.randn(g, C, T) / T ** 0.5, Hh.randn(g, B, C, T)]
    gy = Hh.randn(g, B, C, T)
    x64 = [x.double().requires_grad_(True) for x in xs]
    want = O.timex_conv(*x64, 0.1)
    want = [want.detach()] + list(torch.autograd.grad(want, x64, gy.double()))
    xd = [x.cuda().requires_grad_(True) for x in xs]
    got = R.functions.TimeX.apply(*xd, B, C, T, 0.1)
    got = [got.detach()] + list(torch.autograd.grad(got, xd, gy.cuda()))
    for a, b, name in zip(got, want, ("x", "gw", "gk")):
        Hh.assert_close(a, b, Hh.TOL_FP32_STRICT, f"conv1d {name}")


@pytest.mark.parametrize("T", [72, 100, 160, 256, 257, 300, 768])
def test_errors_of_a_running_sum(T):
    """Whichever form a length takes, it is no further from fp64 than a running fp32 sum of T products: 1.48e-8 sqrt(T) of the norm
    (its partial sums grow as sqrt(t) and each is rounded once); 64 x 8 rows leave 5 % for the draw."""
    import rwkv_cuda_b200 as R
    g = Hh.gen(T)
    B, C = 8, 64
    xs = [Hh.randn(g, C, T) / T ** 0.5, Hh.randn(g, B, C, T)]
    gy = Hh.randn(g, B, C, T)
    x64 = [x.double().requires_grad_(True) for x in xs]
    want = O.timex_conv(*x64, 0.0)
    want = [want.detach(), torch.autograd.grad(want, x64, gy.double())[1]]
    xd = [x.cuda().requires_grad_(True) for x in xs]
    got = R.functions.TimeX.apply(*xd, B, C, T, 0.0)
    got = [got.detach(), torch.autograd.grad(got, xd, gy.cuda())[1]]
    for a, b, name in zip(got, want, ("x", "gk")):
        e = ((a.double().cpu() - b).norm() / b.norm()).item()
        assert e <= 1.05 * 1.48e-8 * T ** 0.5, f"{name}: {e:.3e}"
