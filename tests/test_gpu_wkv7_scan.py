"""GPU parity of RWKV-7 training with the chunks in parallel (few units), against the fp64 oracle: whole and ragged last
chunks, more chunks than records in flight, with and without states; and against the chunk-by-chunk kernels on the same inputs."""
import pytest
import torch

from tests import helpers as Hh

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
NAMES = ("r", "w", "k", "v", "a", "b")


def run(inp, B, T, H, form):
    import rwkv_cuda_b200 as R
    F = R.functions
    xs = [inp[n].to(BF).cuda().view(B, T, H, 64).requires_grad_(True) for n in NAMES]
    s0 = inp["s0"].cuda().requires_grad_(True)
    dy, dsT = inp["dy"].to(BF).cuda(), inp["dsT"].cuda()
    if form == "passing":
        y, sT = F.RWKV7_STATE_PASSING_CLAMPW_CUDA_OP.apply(s0, *xs)
        g = torch.autograd.grad([y, sT], xs + [s0], [dy, dsT])
    elif form == "state":
        y, sT = F.RWKV7_STATE_CLAMPW_CUDA_OP.apply(s0, *xs), None
        g = torch.autograd.grad(y, xs + [s0], dy.view_as(y))
    else:
        y, sT = F.RWKV7_CLAMPW_CUDA_OP.apply(*xs), None
        g = torch.autograd.grad(y, xs, dy.view_as(y))
    assert R._lib.lib().rwkvb200_device_status() == 0
    out = {"y": y.detach().view(B, T, H * 64), **dict(zip(["d" + n for n in NAMES + ("s0",)], g))}
    if sT is not None:
        out["sT"] = sT.detach()
    return out


@pytest.mark.parametrize("form", ["passing", "state", "none"])
@pytest.mark.parametrize("B,T,H", [(1, 80, 1), (2, 96, 3), (1, 272, 2), (3, 128, 5)])
def test_chunks_in_parallel(B, T, H, form):
    import rwkv_cuda_b200 as R
    assert R._lib.lib().rwkvb200_wkv7_train_path(1, B, T, H, 64) == 1
    inp = Hh.v7_inputs(B, T, H, 64, seed=T)
    x64 = {n: (x.double() if n in ("s0", "dsT") else x.to(BF).double()) for n, x in inp.items()}
    want = Hh.v7_oracle(x64, H, use_s0=form != "none", use_dsT=form == "passing")
    got = run(inp, B, T, H, form)
    for n, t in got.items():
        m, e = Hh.assert_close(t, want[n], Hh.TOL_BF16, f"{form} {n}")
        if n in ("sT", "ds0"):
            assert e < 6e-4, (n, e)


def test_agrees_with_the_chunk_by_chunk_kernels():
    import rwkv_cuda_b200 as R
    L = R._lib.lib()
    B, T, H = 2, 1040, 3
    inp = Hh.v7_inputs(B, T, H, 64, seed=1)
    got = run(inp, B, T, H, "passing")
    try:
        assert L.rwkvb200_wkv7_select_form(2) == 0 and L.rwkvb200_wkv7_train_path(1, B, T, H, 64) == 0
        want = run(inp, B, T, H, "passing")
    finally:
        L.rwkvb200_wkv7_select_form(0)
    for n, t in got.items():
        Hh.assert_close(t, want[n].double().cpu(), 1e-2, n)


@pytest.mark.parametrize("form", ["plain", "state", "passing"])
def test_without_tensor_maps(form):
    """Where no tensor maps can be made the forward of the parallel form refuses with nothing enqueued, and the classes take the
    kernels that do without."""
    import rwkv_cuda_b200 as R
    from rwkv_cuda_b200 import _lib
    B, T, H = 2, 160, 2
    inp = Hh.v7_inputs(B, T, H, 64, seed=8)
    assert _lib.lib().rwkvb200_wkv7_train_path(1, B, T, H, 64) == 1
    want = run(inp, B, T, H, form)
    try:
        _lib.call("rwkvb200_test_disable_tensor_maps", 1)
        got = run(inp, B, T, H, form)
    finally:
        _lib.call("rwkvb200_test_disable_tensor_maps", 0)
    for n, t in got.items():
        Hh.assert_close(t, want[n].double().cpu(), 1e-2, n)
