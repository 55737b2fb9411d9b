"""GPU parity of the RWKV-7 inference kernels (head size 64, fp32 arithmetic) against the fp64 oracle at the lengths and
unit counts where their forms change: one token, parts of a step of four tokens, 1, 2 or 4 blocks per unit (16, 16 and 32 tokens staged at
a time), and five stages and more, in which both buffers are handed back."""
import pytest
import torch

from oracle import wkv_oracle as O
from tests import helpers as Hh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,T,H", [(3, 1, 5), (1, 2, 3), (2, 15, 3), (1, 17, 38), (2, 33, 2), (3, 47, 37), (1, 173, 3), (1, 87, 40), (3, 87, 37)])
def test_state_update(dtype, B, T, H):
    import rwkv_cuda_b200 as R
    N, names = 64, ("r", "w", "k", "v", "a", "b")
    inp = Hh.v7_inputs(B, T, H, N, seed=T)
    y64, sT64 = O.wkv7(*(inp[n].to(dtype).double() for n in names), H, s0=inp["s0"].double())
    state = inp["s0"].cuda()
    y = torch.full((B, T, H, N), float("nan"), dtype=dtype, device="cuda")
    R.ops.wkv7_state_update(state, *(inp[n].to(dtype).cuda().view(B, T, H, N).contiguous() for n in names), y)
    Hh.assert_close(y.view(B, T, H * N), y64, Hh.tol_for(dtype), "y")
    Hh.assert_close(state, sT64, 1e-5, "state")   # fp32 whatever the activations are


@pytest.mark.parametrize("name", ["r", "w", "k", "v", "a", "b"])
@pytest.mark.parametrize("t", [4, 6, 7])   # first, third and last token of a step of four
def test_values_that_are_not_finite_stay_behind(t, name):
    """Tokens before such a value, in its own step too, and the rows of other units are those of the call without it."""
    import rwkv_cuda_b200 as R
    B, T, H, N = 1, 17, 2, 64
    inp = Hh.v7_inputs(B, T, H, N, seed=2)

    def call(x):
        state = x["s0"].cuda()
        y = torch.empty(B, T, H, N, device="cuda")
        R.ops.wkv7_state_update(state, *(x[n].float().cuda().view(B, T, H, N).contiguous() for n in ("r", "w", "k", "v", "a", "b")), y)
        return y, state

    y0, s0 = call(inp)
    bad = dict(inp)
    bad[name] = inp[name].clone().reshape(B, T, H, N)
    bad[name][0, t, 0, 5] = float("nan")
    y, s = call(bad)
    assert torch.equal(y[:, :t], y0[:, :t]) and torch.equal(y[:, :, 1], y0[:, :, 1]) and torch.equal(s[:, 1], s0[:, 1])
    assert torch.isnan(y[:, t:, 0]).any()


def test_errors_of_a_prompt():
    """The state against fp64 is no further off than with one token as a step (S_t = (S_{t-1} d_t + k_t v_t) + sa_t b_t, each multiply-add
    rounded once) and the same fp32 decays; 2 % for the sample of 32768 elements."""
    import rwkv_cuda_b200 as R
    T, H, N, names = 203, 8, 64, ("r", "w", "k", "v", "a", "b")
    inp = Hh.v7_inputs(1, T, H, N, seed=11)
    x = [inp[n].view(1, T, H, N).cuda() for n in names]
    state, y = inp["s0"].cuda(), torch.empty(1, T, H, N, device="cuda")
    R.ops.wkv7_state_update(state, *x, y)
    # a state of ones and no other input: the decays as the kernel has them
    ones, zero = torch.ones(T, H, N, N, device="cuda"), torch.zeros(T, 1, H, N, device="cuda")
    R.ops.wkv7_state_update(ones, zero, x[1].transpose(0, 1).contiguous(), zero, zero, zero, zero, torch.empty_like(zero))
    d32 = ones[:, :, 0].double().cpu()
    r, w, k, v, a, b = (inp[n].view(T, H, N).double() for n in names)
    d64, fl = torch.exp(-0.6065306597126334 * torch.sigmoid(w)), lambda z: z.float().double()
    exact, S = inp["s0"][0].double(), inp["s0"][0].double()
    sa = fl((S * a[0][:, None]).sum(2))
    for t in range(T):
        exact = exact * d64[t][:, None] + (exact * a[t][:, None]).sum(2)[..., None] * b[t][:, None] + v[t][..., None] * k[t][:, None]
        G = fl(S * d32[t][:, None] + fl(v[t][..., None] * k[t][:, None]))
        S = fl(G + sa[..., None] * b[t][:, None])
        if t + 1 < T:
            sa = fl(sa * fl((b[t] * a[t + 1]).sum(1))[:, None] + fl((G * a[t + 1][:, None]).sum(2)))
    error = lambda z: ((z - exact).norm() / exact.norm()).item()
    assert error(state[0].double().cpu()) <= 1.02 * error(S), (error(state[0].double().cpu()), error(S))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("name", ["r", "k", "v", "a", "b", "s0"])
@pytest.mark.parametrize("H", [2, 40, 80])   # four, two blocks and one per unit
def test_infinities_of_the_recurrence(H, name, value, dtype):
    """Infinities, NaN and numbers stand where the recurrence has them token by token (S_t = G_t + sa_t b_t with G_t = S_{t-1} d_t + v_t k_t,
    sa_{t+1} = G_t.a_{t+1} + sa_t (b_t.a_{t+1})): in what order a sum over keys is taken does not change that."""
    import rwkv_cuda_b200 as R
    B, T, N, t, names = 1, 11, 64, 6, ("r", "w", "k", "v", "a", "b")
    inp = {n: x.clone().reshape(B, T, H, N) if x.dim() == 3 else x.clone() for n, x in Hh.v7_inputs(B, T, H, N, seed=4).items()}
    if name == "s0":
        inp["s0"][0, 0, 3, 5] = value
    else:
        inp[name][0, t, 0, 5] = value
    x = [inp[n].to(dtype).cuda().contiguous() for n in names]
    state, y = inp["s0"].cuda(), torch.empty(B, T, H, N, dtype=dtype, device="cuda")
    R.ops.wkv7_state_update(state, *x, y)

    r, w, k, v, a, b = (inp[n][0, :, 0].to(dtype).double() for n in names)
    d, S, rows = torch.exp(-0.6065306597126334 * torch.sigmoid(w)), inp["s0"][0, 0].double(), []
    sa = (S * a[0]).sum(1)
    for i in range(T):
        G = S * d[i] + v[i][:, None] * k[i]
        S = G + sa[:, None] * b[i]
        rows.append((S * r[i]).sum(1))
        if i + 1 < T:
            sa = (G * a[i + 1]).sum(1) + sa * (b[i] * a[i + 1]).sum()
    for got, want in ((y[0, :, 0], torch.stack(rows)), (state[0, 0], S)):
        got = got.double().cpu()
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isposinf(), want.isposinf()) and torch.equal(got.isneginf(), want.isneginf())
        ok = want.isfinite()
        assert not ok.any() or (got[ok] - want[ok]).abs().max() <= Hh.tol_for(dtype) * want[ok].abs().max()
