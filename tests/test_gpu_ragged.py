"""GPU parity at sequence lengths that are not whole chunks: the tensor-core kernels of RWKV-5 and RWKV-6 mask the tokens
of a partial 32-token chunk.  Against the fp64 oracle, through the training classes."""
import pytest
import torch

from oracle import wkv_oracle as O
from tests import helpers as Hh

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def grads(fn, tensors, gy, dev=None):
    xs = [(x.to(BF).to(dev) if dev else x.to(BF).double()).requires_grad_(True) for x in tensors]
    y = fn(*xs)
    return [y.detach()] + list(torch.autograd.grad(y, xs, gy.to(BF).to(dev) if dev else gy.to(BF).double()))


@pytest.mark.parametrize("op", ["wkv5", "wkv6", "wkv6 strong decay"])
@pytest.mark.parametrize("B,T,H", [(3, 31, 1), (1, 33, 1), (3, 47, 2), (2, 65, 3), (2, 191, 2)])
def test_training_at_any_length(op, B, T, H):
    import rwkv_cuda_b200 as R
    g = Hh.gen(T)
    N, C = 64, H * 64
    r, k, v = (0.5 * Hh.randn(g, B, T, C) for _ in range(3))
    u, gy = Hh.rand(g, H, N, lo=-1, hi=1), Hh.randn(g, B, T, C)
    if op == "wkv5":
        w = Hh.rand(g, H, N, lo=-6, hi=-1)
        ours, oracle = R.functions.WKV_5, O.wkv5
    else:
        w = Hh.randn(g, B, T, C) + (2.0 if "strong" in op else -3.0)
        ours, oracle = R.functions.WKV_6, O.wkv6
    got = grads(lambda *xs: ours.apply(B, T, C, H, *xs), (r, k, v, w, u), gy, "cuda")
    want = grads(lambda *xs: oracle(*xs, H), (r, k, v, w, u), gy)
    for a, b, name in zip(got, want, ("y", "gr", "gk", "gv", "gw", "gu")):
        Hh.assert_close(a, b, Hh.TOL_BF16, f"{op} {name}")
