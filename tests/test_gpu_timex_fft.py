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
