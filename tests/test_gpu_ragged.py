"""GPU parity at sequence lengths that are not whole chunks, against the fp64 oracle, through the training classes.  RWKV-5 and
RWKV-6 compute them in fp32, split over time into segments of 32 tokens."""
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


@pytest.mark.parametrize("op", ["wkv5", "wkv6"])
@pytest.mark.parametrize("B,T,H", [(2, 33, 1), (1, 47, 3), (2, 191, 2), (1, 1000, 2)])
def test_fp32_arithmetic_where_T_is_ragged(op, B, T, H):
    """Every output is one rounding to bf16 away from fp64 (2^-8 of the value at most; TF32 operands add a few 2^-11 of the output's
    size), and fp32 sums over at most 1000 tokens of 64 keys add less than 2^-15 of it."""
    import rwkv_cuda_b200 as R
    g = Hh.gen(T)
    N, C = 64, H * 64
    r, k, v = (0.5 * Hh.randn(g, B, T, C) for _ in range(3))
    u, gy = Hh.rand(g, H, N, lo=-1, hi=1), Hh.randn(g, B, T, C)
    w = Hh.rand(g, H, N, lo=-6, hi=-1) if op == "wkv5" else Hh.randn(g, B, T, C) - 5.0
    ours, oracle = (R.functions.WKV_5, O.wkv5) if op == "wkv5" else (R.functions.WKV_6, O.wkv6)
    got = grads(lambda *xs: ours.apply(B, T, C, H, *xs), (r, k, v, w, u), gy, "cuda")
    want = grads(lambda *xs: oracle(*xs, H), (r, k, v, w, u), gy)
    for a, b, name in zip(got, want, ("y", "gr", "gk", "gv", "gw", "gu")):
        size = torch.maximum(b.abs(), b.square().mean().sqrt())
        err = ((a.double().cpu().reshape(b.shape) - b).abs() / size).max().item()
        assert err <= 2 ** -8 + 2 ** -15, f"{op} {name}: {err:.3e}"


@pytest.mark.parametrize("use_s0", [False, True])
def test_rwkv7_training_classes(use_s0):
    import rwkv_cuda_b200 as R
    B, T, H, N = 2, 48, 2, 64
    inp = Hh.v7_inputs(B, T, H, N, seed=3)
    names = ("r", "w", "k", "v", "a", "b")
    x64 = {n: (x.double() if n in ("s0", "dsT") else x.to(BF).double()) for n, x in inp.items()}
    want = Hh.v7_oracle(x64, H, use_s0=use_s0, use_dsT=False)
    xs = [inp[n].to(BF).cuda().requires_grad_(True) for n in names]
    s0 = inp["s0"].cuda().requires_grad_(True)
    y = R.functions.RWKV7_STATE_CLAMPW_CUDA(s0, *xs) if use_s0 else R.functions.RWKV7_CLAMPW_CUDA(*xs)
    g = torch.autograd.grad(y, xs + ([s0] if use_s0 else []), inp["dy"].to(BF).cuda())
    Hh.assert_close(y, want["y"], Hh.TOL_BF16, "y")
    for a, n in zip(g, names + ("s0",)):
        Hh.assert_close(a, want["d" + n], Hh.TOL_BF16, "d" + n)


@pytest.mark.parametrize("T", [64, 300])
@pytest.mark.parametrize("shift", [-5.0, -1.5, -0.5])
def test_rwkv6_forward_scales_its_state(shift, T):
    """Decays with which the forward scales the state in tensor memory never, every few chunks and before every chunk."""
    import rwkv_cuda_b200 as R
    g = Hh.gen(7)
    B, H, N = 2, 2, 64
    C = H * N
    r, k, v = (0.5 * Hh.randn(g, B, T, C) for _ in range(3))
    w, u, s0 = Hh.randn(g, B, T, C) + shift, Hh.rand(g, H, N, lo=-1, hi=1), 0.1 * Hh.randn(g, B, H, N, N)
    yo, sTo = O.wkv6(*(x.to(BF).double() for x in (r, k, v, w, u)), H, s0=s0.double(), return_state=True)
    d = [x.to(BF).to("cuda").contiguous() for x in (r, k, v, w, u)]
    y, sT = torch.full((B, T, C), float("nan"), dtype=BF, device="cuda"), torch.full((B, H, N, N), float("nan"), device="cuda")
    R.ops.wkv6state_forward_ex(B, T, C, H, *d, s0.to("cuda"), y, sT)
    Hh.assert_close(y, yo, Hh.TOL_BF16, "y")
    Hh.assert_close(sT, sTo, Hh.TOL_BF16, "sT")


# few segments; enough of them for the products, with states by a walk along the segments and (32 units) by a scan over them
@pytest.mark.parametrize("B,T,H", [(1, 71, 2), (5, 33, 64), (3, 47, 110), (2, 333, 40), (1, 1000, 32)])
def test_rwkv6_segments_of_both_kinds(B, T, H):
    """Segments with decays too strong for the matrix form (or for its anchor in the middle) beside others, every tensor one element off
    its alignment: bounds as above."""
    import rwkv_cuda_b200 as R
    g = Hh.gen(T)
    N, C = 64, H * 64
    r, k, v = (0.5 * Hh.randn(g, B, T, C) for _ in range(3))
    u, gy, w = Hh.rand(g, H, N, lo=-1, hi=1), Hh.randn(g, B, T, C), Hh.randn(g, B, T, C) - 4.0
    w[:, -7, 3] = 6.0             # one token of a segment, one channel
    w[:, 64:, 2 * 64 - 1] = 1.5   # exp(1.5) * 16 > 60: from the third segment on
    odd = lambda x: torch.cat([x.new_zeros(1), x.flatten()]).to(BF).cuda()[1:].view(x.shape)
    xs = [odd(x).requires_grad_(True) for x in (r, k, v, w, u)]
    y = R.functions.WKV_6.apply(B, T, C, H, *xs)
    got = [y, *torch.autograd.grad(y, xs, odd(gy))]
    xo = [x.to(BF).double().requires_grad_(True) for x in (r, k, v, w, u)]
    yo = O.wkv6(*xo, H)
    want = [yo, *torch.autograd.grad(yo, xo, gy.to(BF).double())]
    for a, b, name in zip(got, want, ("y", "gr", "gk", "gv", "gw", "gu")):
        size = torch.maximum(b.abs(), b.square().mean().sqrt())
        err = ((a.double().cpu().reshape(b.shape) - b).abs() / size).max().item()
        assert err <= 2 ** -8 + 2 ** -15, f"{name}: {err:.3e}"


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("name", ["v", "k", "r"])
def test_rwkv6_values_that_are_not_finite_stay_behind(name, value):
    """Tokens before such a value are those of the call without it, inside its segment too."""
    import rwkv_cuda_b200 as R
    B, T, H, N, t = 1, 71, 220, 64, 45   # (more than four segments per SM: by products)
    g = Hh.gen(5)
    C = H * N
    x = {n: 0.5 * Hh.randn(g, B, T, C) for n in ("r", "k", "v")}
    w, u = Hh.randn(g, B, T, C) - 4.0, Hh.rand(g, H, N, lo=-1, hi=1)
    call = lambda: R.functions.WKV_6.apply(B, T, C, H, *(a.to(BF).cuda() for a in (x["r"], x["k"], x["v"], w, u)))
    clean = call()
    x[name][:, t, 7] = value
    y = call()
    size = clean.float().square().mean().sqrt()
    assert ((y[:, :t].float() - clean[:, :t].float()).abs() / size).max().item() < 2 ** -6   # (other kernel: other rounding, in bf16)
    assert not torch.isfinite(y[:, t]).all()


@pytest.mark.parametrize("B,T,H", [(5, 40, 64), (2, 333, 40), (1, 1000, 32)])
def test_rwkv5_fp32_by_products(B, T, H):
    """fp32 through the products of split operands, heads with decays too strong for them among the others, tensors off their alignment.
    Bounds: a sum of n products has an error of about sqrt(n) 2^-24 of their size; n is at most 64 keys x some 32 tokens, and gw
    weights its terms by their distance in time (test of the operator: 1e-4)."""
    import rwkv_cuda_b200 as R
    g = Hh.gen(T)
    N, C = 64, H * 64
    r, k, v = (0.5 * Hh.randn(g, B, T, C) for _ in range(3))
    u, gy, w = Hh.rand(g, H, N, lo=-1, hi=1), Hh.randn(g, B, T, C), Hh.rand(g, H, N, lo=-6, hi=-1)
    w[1, 5], w[2] = 2.0, 1.0
    odd = lambda x: torch.cat([x.new_zeros(1), x.flatten()]).float().cuda()[1:].view(x.shape)
    xs = [odd(x).requires_grad_(True) for x in (r, k, v, w, u)]
    y = R.functions.WKV_5.apply(B, T, C, H, *xs)
    got = [y, *torch.autograd.grad(y, xs, odd(gy))]
    xo = [x.float().double().requires_grad_(True) for x in (r, k, v, w, u)]
    yo = O.wkv5(*xo, H)
    want = [yo, *torch.autograd.grad(yo, xo, gy.float().double())]
    for a, b, name in zip(got, want, ("y", "gr", "gk", "gv", "gw", "gu")):
        err = ((a.double().cpu().reshape(b.shape) - b).norm() / b.norm()).item()
        assert err <= 1e-6, f"{name}: {err:.3e}"


# states by a walk along the segments (more than a unit per two SMs) and by a scan over them; products and (1, 40, 3) token by token
@pytest.mark.parametrize("B,T,H,dtype", [(5, 40, 64, torch.float32), (2, 333, 40, BF), (1, 1000, 32, torch.float32), (1, 40, 3, torch.float32)])
@pytest.mark.parametrize("w0", [95.0, 88.5, 20.0])
def test_rwkv5_decay_of_zero(w0, B, T, H, dtype):
    """exp(-exp(w0)) is 0 and (above 88.3) its logarithm -inf: a token reaches the next one only.  Bounds as above; dL/dw of such a
    channel is -inf * 0 in fp32 and is left out."""
    import rwkv_cuda_b200 as R
    g = Hh.gen(T)
    N, C = 64, H * 64
    r, k, v = (0.5 * Hh.randn(g, B, T, C) for _ in range(3))
    u, gy, w = Hh.rand(g, H, N, lo=-1, hi=1), Hh.randn(g, B, T, C), Hh.rand(g, H, N, lo=-6, hi=-1)
    w[1, 5] = w[2, 63] = w0
    xs = [x.to(dtype).cuda().requires_grad_(True) for x in (r, k, v, w, u)]
    y = R.functions.WKV_5.apply(B, T, C, H, *xs)
    got = [y, *torch.autograd.grad(y, xs, gy.to(dtype).cuda())]
    xo = [x.to(dtype).double().requires_grad_(True) for x in (r, k, v, w, u)]
    yo = O.wkv5(*xo, H)
    want = [yo, *torch.autograd.grad(yo, xo, gy.to(dtype).double())]
    for a, b, name in zip(got, want, ("y", "gr", "gk", "gv", "gw", "gu")):
        a = a.detach().double().cpu().reshape(b.shape)
        if name == "gw":
            a, b = (torch.where(w == w0, torch.zeros_like(x), x) for x in (a, b))
        if dtype == BF:
            err = ((a - b).abs() / torch.maximum(b.abs(), b.square().mean().sqrt())).max().item()
            assert err <= 2 ** -8 + 2 ** -15, f"{name}: {err:.3e}"
        else:
            err = ((a - b).norm() / b.norm()).item()
            assert err <= 2e-6, f"{name}: {err:.3e}"


@pytest.mark.parametrize("name", ["gy", "k", "r"])
def test_rwkv6_products_that_overflow(name):
    """Decays just inside the range of the matrix form and a tensor of 1e20: scaled operands times it leave fp32's range, the results do
    not.  Bounds as above."""
    import rwkv_cuda_b200 as R
    B, T, H, N = 2, 333, 40, 64
    g = Hh.gen(1)
    C = H * N
    x = {n: 0.5 * Hh.randn(g, B, T, C) for n in ("r", "k", "v", "gy")}
    x[name] *= 1e20
    w, u = Hh.randn(g, B, T, C) - 5.0, Hh.rand(g, H, N, lo=-1, hi=1)
    w.view(B, T, H, N)[..., 9] = 1.2   # 16 exp(1.2) log2(e) = 77
    xs = [a.to(BF).cuda().requires_grad_(True) for a in (x["r"], x["k"], x["v"], w, u)]
    y = R.functions.WKV_6.apply(B, T, C, H, *xs)
    got = [y, *torch.autograd.grad(y, xs, x["gy"].to(BF).cuda())]
    xo = [a.to(BF).double().requires_grad_(True) for a in (x["r"], x["k"], x["v"], w, u)]
    yo = O.wkv6(*xo, H)
    want = [yo, *torch.autograd.grad(yo, xo, x["gy"].to(BF).double())]
    for a, b, name in zip(got, want, ("y", "gr", "gk", "gv", "gw", "gu")):
        size = torch.maximum(b.abs(), b.square().mean().sqrt())
        err = ((a.double().cpu().reshape(b.shape) - b).abs() / size).max().item()
        assert err <= 2 ** -8 + 2 ** -15, f"{name}: {err:.3e}"


@pytest.mark.parametrize("shift", [-10.0, -5.0])
def test_rwkv6_states_of_the_walk(shift):
    """fp32 states at the start of every segment (left for the backward), with slow decays: sums over the whole sequence.  Bound: one rounding
    per segment at the size of the state, 32 of them at random, and four at the size of a segment's own sum, all 2^-24."""
    import rwkv_cuda_b200 as R
    B, T, H, N = 2, 1000, 40, 64   # (more than a unit per two SMs: by the walk)
    g = Hh.gen(3)
    C, nseg = H * N, (T + 31) // 32
    r, k, v = (0.5 * Hh.randn(g, B, T, C) for _ in range(3))
    w, u = Hh.randn(g, B, T, C) + shift, Hh.rand(g, H, N, lo=-1, hi=1)
    d = [x.to(BF).cuda() for x in (r, k, v, w, u)]
    y = torch.empty_like(d[0])
    saved = torch.empty(R._lib.lib().rwkvb200_wkv6_train_saved_bytes(R._lib.BF16, B, T, C, H) // 4 + 1, device="cuda")
    rc = R._lib.lib().rwkvb200_wkv6_train_forward(R._lib.BF16, B, T, C, H, *(x.data_ptr() for x in d), None, y.data_ptr(), None, saved.data_ptr(),
                                                  torch.cuda.current_stream().cuda_stream)
    assert rc == 2, rc
    got = saved[:B * H * nseg * N * N].view(B, H, nseg, N, N).double()
    kk, vv, dd = (x.double().view(B, T, H, N) for x in (d[1], d[2], torch.exp(-torch.exp(d[3].double()))))
    S = torch.zeros(B, H, N, N, dtype=torch.float64, device="cuda")
    err = size = 0.0
    for t in range(T):
        if t % 32 == 0:
            err, size = err + (got[:, :, t // 32] - S).square().sum().item(), size + S.square().sum().item()
        S = S * dd[:, t, :, :, None] + kk[:, t, :, :, None] * vv[:, t, :, None, :]
    assert (err / size) ** 0.5 <= (32 ** 0.5 + 4) * 2 ** -24, (err / size) ** 0.5


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("name", ["r", "k", "v", "gy"])
@pytest.mark.parametrize("op", ["wkv6", "wkv5 fp32"])
def test_values_that_are_not_finite_as_token_by_token(op, name, value):
    """y and gradients of two heads in a call with many heads (states by the walk, the rest by products) and in one with these two only
    (token by token): infinities, NaN and numbers in the same places."""
    import rwkv_cuda_b200 as R
    B, T, N, t, H = 1, 103, 64, 45, 160
    dtype, F = (BF, R.functions.WKV_6) if op == "wkv6" else (torch.float32, R.functions.WKV_5)
    g = Hh.gen(5)
    x = {n: 0.5 * Hh.randn(g, B, T, H, N) for n in ("r", "k", "v", "gy")}
    x["w"] = Hh.randn(g, B, T, H, N) - 4.0 if op == "wkv6" else Hh.rand(g, H, N, lo=-6, hi=-1)
    x["u"] = Hh.rand(g, H, N, lo=-1, hi=1)
    x[name][:, t, 0, 7] = value

    def call(H):
        xs = [(x[n][:, :, :H].reshape(B, T, H * N) if x[n].dim() == 4 else x[n][:H]).to(dtype).cuda().contiguous().requires_grad_(n != "gy")
              for n in ("r", "k", "v", "w", "u", "gy")]
        y = F.apply(B, T, H * N, H, *xs[:5])
        out = [y, *torch.autograd.grad(y, xs[:5], xs[5])]
        return [(z.view(B, T, H, N)[:, :, :2] if z.dim() == 3 else z.view(H, N)[:2]).float() for z in out]

    for a, b, out in zip(call(H), call(2), ("y", "gr", "gk", "gv", "gw", "gu")):
        assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isposinf(), b.isposinf()) and torch.equal(a.isneginf(), b.isneginf()), out
        a, b = (torch.where(z.isfinite(), z, torch.zeros_like(z)) for z in (a, b))
        assert ((a - b).abs() / torch.maximum(b.abs(), b.square().mean().sqrt())).max().item() <= (2 ** -7 if dtype == BF else 2e-5), out


@pytest.mark.parametrize("B,T,H", [(2, 333, 40), (1, 1000, 32)])
@pytest.mark.parametrize("lo,hi", [(-6.0, -5.0), (-2.0, -1.5), (-1.2, -1.0)])
def test_rwkv5_fp32_decay_gradient(lo, hi, B, T, H):
    """All channels decay alike, so that none hides behind a slower one.  Bound of gw: a sum over tokens of sums over tokens, keys and values,
    each with an error of a few 2^-24 of its size at random: 10 2^-24 (token by token 4.8 at w around -1.1, 16 around -5.5)."""
    import rwkv_cuda_b200 as R
    g = Hh.gen(T)
    N, C = 64, H * 64
    r, k, v = (0.5 * Hh.randn(g, B, T, C) for _ in range(3))
    u, gy, w = Hh.rand(g, H, N, lo=-1, hi=1), Hh.randn(g, B, T, C), Hh.rand(g, H, N, lo=lo, hi=hi)
    xs = [x.cuda().requires_grad_(True) for x in (r, k, v, w, u)]
    y = R.functions.WKV_5.apply(B, T, C, H, *xs)
    got = torch.autograd.grad(y, xs, gy.cuda())
    xo = [x.double().requires_grad_(True) for x in (r, k, v, w, u)]
    want = torch.autograd.grad(O.wkv5(*xo, H), xo, gy.double())
    for a, b, name in zip(got, want, ("gr", "gk", "gv", "gw", "gu")):
        err = ((a.double().cpu().reshape(b.shape) - b).norm() / b.norm()).item()
        assert err <= 10 * 2 ** -24, f"{name}: {err:.3e}"


@pytest.mark.parametrize("lo,hi", [(-6.0, -1.0), (-3.0, -2.5), (-0.6, -0.4)])
def test_rwkv5_fp32_errors(lo, hi):
    """y and gradients by products, a few 2^-24 of their norm (-0.6 to -0.4, just inside the limit of these kernels: token by token 1.5 2^-24;
    powers of a decay as exponentials of a rounded product 2.5).  -6 to -1: sums over the slow channels' long memory, token by token 8.7."""
    import rwkv_cuda_b200 as R
    B, T, H, N = 2, 333, 40, 64
    g = Hh.gen(T)
    C = H * N
    r, k, v = (0.5 * Hh.randn(g, B, T, C) for _ in range(3))
    u, gy, w = Hh.rand(g, H, N, lo=-1, hi=1), Hh.randn(g, B, T, C), Hh.rand(g, H, N, lo=lo, hi=hi)
    xs = [x.cuda().requires_grad_(True) for x in (r, k, v, w, u)]
    y = R.functions.WKV_5.apply(B, T, C, H, *xs)
    got = [y, *torch.autograd.grad(y, xs, gy.cuda())]
    xo = [x.double().requires_grad_(True) for x in (r, k, v, w, u)]
    yo = O.wkv5(*xo, H)
    want = [yo, *torch.autograd.grad(yo, xo, gy.double())]
    for a, b, name in list(zip(got, want, ("y", "gr", "gk", "gv")))[:4]:
        err = ((a.double().cpu().reshape(b.shape) - b).norm() / b.norm()).item()
        assert err <= (2.2 if hi > -1 else 3) * 2 ** -24, f"{name}: {err:.3e}"


@pytest.mark.parametrize("T", [34, 48, 64, 65])
def test_rwkv5_segments_left_to_the_other_kernel(T):
    """A head with a channel that decays by more than a factor of 2 per token is left to the token-by-token kernels, its last segment too however
    short, and no other head."""
    import rwkv_cuda_b200 as R
    B, H, N = 5, 64, 64
    g = Hh.gen(T)
    C, nseg = H * N, (T + 31) // 32
    d = [(0.5 * Hh.randn(g, B, T, C)).cuda() for _ in range(3)]
    w, u = Hh.rand(g, H, N, lo=-6, hi=-0.4), Hh.rand(g, H, N, lo=-1, hi=1)
    w[3, 5], w[60, 63] = 1.0, -0.3
    y = torch.empty_like(d[0])
    lib, n = R._lib.lib(), B * H * nseg
    saved = torch.empty(lib.rwkvb200_wkv5_train_saved_bytes(B, T, C, H) // 4, dtype=torch.int32, device="cuda")
    rc = lib.rwkvb200_wkv5_train_forward(R._lib.F32, B, T, C, H, *(x.data_ptr() for x in (*d, w.cuda(), u.cuda(), y)), saved.data_ptr(),
                                         torch.cuda.current_stream().cuda_stream)
    assert rc == 1, rc
    flags = saved[n * N * N:n * N * N + n].view(B, H, nseg).bool().cpu()
    want = torch.zeros_like(flags)
    want[:, [3, 60]] = True
    assert torch.equal(flags, want)


@pytest.mark.parametrize("w0", [0.72, 0.74, 1.3, 1.4])   # inside and outside of 48 bits up to the middle of a segment, and of 86
@pytest.mark.parametrize("scale", [1e-14, 1e-8, 1e12])
def test_rwkv6_gradients_of_any_size(scale, w0):
    """One channel with a strong decay beside others, gradients that a loss scale made large or small; the gradients of that channel by
    themselves.  Bounds as above."""
    import rwkv_cuda_b200 as R
    B, T, H, N = 2, 333, 40, 64
    g = Hh.gen(1)
    C = H * N
    r, k, v = (0.5 * Hh.randn(g, B, T, C) for _ in range(3))
    gy, w, u = scale * Hh.randn(g, B, T, C), Hh.randn(g, B, T, C) - 5.0, Hh.rand(g, H, N, lo=-1, hi=1)
    w.view(B, T, H, N)[..., 9] = w0
    xs = [a.to(BF).cuda().requires_grad_(True) for a in (r, k, v, w, u)]
    y = R.functions.WKV_6.apply(B, T, C, H, *xs)
    got = [y, *torch.autograd.grad(y, xs, gy.to(BF).cuda())]
    xo = [a.to(BF).double().requires_grad_(True) for a in (r, k, v, w, u)]
    yo = O.wkv6(*xo, H)
    want = [yo, *torch.autograd.grad(yo, xo, gy.to(BF).double())]
    for a, b, name in zip(got, want, ("y", "gr", "gk", "gv", "gw", "gu")):
        a, b = (z.detach().double().cpu().reshape(-1, N) for z in (a, b))
        for part in (slice(0, N), slice(9, 10)):
            size = torch.maximum(b[:, part].abs(), b[:, part].square().mean().sqrt())
            err = ((a[:, part] - b[:, part]).abs() / size).max().item()
            assert err <= 2 ** -8 + 2 ** -15, f"{name} {part}: {err:.3e}"


@pytest.mark.parametrize("op,H", [("wkv6", 512), ("wkv5 fp32", 640)])
def test_many_segments_some_left_to_the_other_kernels(op, H):
    """So many segments (7680 and 9600) that a block of the token-by-token kernels looks at several: heads with strong decays, throughout or in a few
    segments, and their neighbours against a call with these heads only (few segments: token by token)."""
    import rwkv_cuda_b200 as R
    B, T, N, picks = 1, 463, 64, [0, 7, 8, 200, 201, H - 1]
    dtype, F = (BF, R.functions.WKV_6) if op == "wkv6" else (torch.float32, R.functions.WKV_5)
    g = torch.Generator(device="cuda").manual_seed(3)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x = {n: 0.5 * rn(B, T, H, N) for n in ("r", "k", "v", "gy")}
    x["u"] = rn(H, N)
    if op == "wkv6":
        x["w"] = rn(B, T, H, N) - 4.0
        x["w"][:, :, 7, 3] = x["w"][:, 40:100, 200, 5] = x["w"][:, -1, H - 1, 0] = 4.0
    else:
        x["w"] = torch.rand(H, N, device="cuda", generator=g) * 5.0 - 6.0
        x["w"][7, 3] = x["w"][200, 5] = x["w"][H - 1, 0] = 2.0

    def call(heads):
        xs = [(x[n][:, :, heads].reshape(B, T, -1) if x[n].dim() == 4 else x[n][heads]).to(dtype).contiguous().requires_grad_(n != "gy")
              for n in ("r", "k", "v", "w", "u", "gy")]
        y = F.apply(B, T, len(heads) * N, len(heads), *xs[:5])
        out = [y, *torch.autograd.grad(y, xs[:5], xs[5])]
        return [z.view(B, T, len(heads), N) if z.dim() == 3 else z.view(len(heads), N) for z in out]

    for a, b, name in zip(call(list(range(H))), call(picks), ("y", "gr", "gk", "gv", "gw", "gu")):
        a = (a[:, :, picks] if a.dim() == 4 else a[picks]).float()
        err = ((a - b.float()).abs() / torch.maximum(b.float().abs(), b.float().square().mean().sqrt())).max().item()
        assert err <= (2 ** -7 if dtype == BF else 2e-5), f"{name}: {err:.3e}"
