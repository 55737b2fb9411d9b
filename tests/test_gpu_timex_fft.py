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


def run(xs, gy, B, C, T):
    import rwkv_cuda_b200 as R
    xd = [x.cuda().requires_grad_(True) for x in xs]
    got = R.functions.TimeX.apply(*xd, B, C, T, 0.1)
    return [x.detach().cpu() for x in (got, *torch.autograd.grad(got, xd, gy.cuda()))]


@pytest.mark.parametrize("T", [300, 768])
def test_rows_keep_their_own_precision(T):
    """Rows of very different sizes side by side, one of zeros among them: every row is exact to its own norm (the tolerance of the
    operator), and zeros stay zeros."""
    g = Hh.gen(T)
    B, C = 7, 2
    size = torch.tensor([1.0, 1e6, 0.0, 3.0, 1e-6, 1e-9, 2.0]).view(B, 1, 1)
    xs = [Hh.randn(g, C, T) / T ** 0.5, Hh.randn(g, B, C, T) * size]
    gy = Hh.randn(g, B, C, T) * size.flip(0)
    x64 = [x.double().requires_grad_(True) for x in xs]
    want = O.timex_conv(*x64, 0.0)
    want = [want.detach()] + list(torch.autograd.grad(want, x64, gy.double()))
    x, gw, gk = run(xs, gy, B, C, T)
    Hh.assert_close(gw, want[1], Hh.TOL_FP32_STRICT, "gw")
    for b in range(B):
        if size[b] >= 1:   # (0.1 is added to the output)
            Hh.assert_close(x[b], want[0][b] + 0.1, Hh.TOL_FP32_STRICT, f"x of row {b}")
        if size[B - 1 - b] > 0:
            Hh.assert_close(gk[b], want[2][b], Hh.TOL_FP32_STRICT, f"gk of row {b}")
    assert (x[2] == 0.1).all() and (gk[B - 3] == 0).all()
    assert (x[5] - 0.1).abs().max() < 1e-7


@pytest.mark.parametrize("bad", [float("inf"), float("nan"), 3e38])
@pytest.mark.parametrize("T", [300, 768])
def test_values_a_transform_cannot_take(T, bad):
    """A value that is not finite, or nearly the largest there is, reaches the tokens that it belongs to and nothing else."""
    g = Hh.gen(T)
    B, C, t0 = 5, 3, T // 3
    xs = [Hh.randn(g, C, T) / T ** 0.5, Hh.randn(g, B, C, T)]
    gy = Hh.randn(g, B, C, T)
    x64 = [x.double().requires_grad_(True) for x in xs]
    want = O.timex_conv(*x64, 0.1)
    want = [want.detach()] + list(torch.autograd.grad(want, x64, gy.double()))
    dirty = [xs[0].clone(), xs[1].clone()]
    dirty[1][2, 0, t0] = bad          # row 2 of channel 0
    dirty[0][1, T - 1 - t0] = bad     # the tap of channel 1 that reaches back t0 tokens
    gd = gy.clone()
    gd[3, 2, t0] = bad                # a gradient of channel 2
    x, gw, gk = run(dirty, gd, B, C, T)
    clean_x, clean_gw, clean_gk = (torch.ones(s, dtype=torch.bool) for s in ((B, C, T), (C, T), (B, C, T)))
    clean_x[2, 0, t0:] = False
    clean_x[:, 1, t0:] = False
    clean_gk[:, 1, :T - t0] = False   # gk[u] takes g of the tokens from u on
    clean_gk[3, 2, :t0 + 1] = False
    clean_gw[0, t0:] = False          # gw[T-1-lag] sums g[t] k[t-lag]: k of token t0 meets the lags up to T-1-t0
    clean_gw[2, T - 1 - t0:] = False  # ... g of token t0 the lags up to t0
    for got, ref, clean, name in zip((x, gw, gk), want, (clean_x, clean_gw, clean_gk), ("x", "gw", "gk")):
        Hh.assert_close(got[clean], ref[clean], Hh.TOL_FP32_STRICT, name)
        assert (~(got[~clean].abs() < 1e30)).float().mean() > 0.9, name


@pytest.mark.parametrize("T", [511, 512, 513, 514, 640, 767, 768, 769])   # both ends of the transforms of 1536 points (513 to 768 tokens)
@pytest.mark.parametrize("B,C", [(1, 2), (3, 2), (33, 2)])
def test_lengths_that_are_three_times_a_power_of_two(B, C, T):
    test_conv1d_training_class(B, C, T)
    test_errors_of_a_running_sum(T)
