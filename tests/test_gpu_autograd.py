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


@pytest.mark.parametrize("name", NAMES)
def test_calls_that_only_an_autograd_function_can_take(name):
    """jit tracing records the operator and not its result; forward-mode derivatives and functorch's transforms are refused and not
    ignored; a subclass may replace forward and backward; and forward and backward give what the native node gives."""
    import torch.autograd.forward_ad as fwAD
    xs, call = cases()[name]
    xs = [x.cuda() for x in xs]
    first = lambda *x: outputs(call(*x))[0]
    traced = torch.jit.trace(first, tuple(xs), check_trace=False)
    other = [x.flip(0).contiguous() for x in xs]
    assert torch.equal(traced(*other), first(*other))
    with fwAD.dual_level(), pytest.raises((NotImplementedError, RuntimeError)):
        call(*(fwAD.make_dual(x, torch.ones_like(x)) for x in xs))
    for transform in (lambda: torch.func.grad(lambda *x: first(*x).float().sum())(*xs), lambda: torch.func.vjp(call, *xs),
                      lambda: torch.vmap(call)(*(torch.stack([x, x]) for x in xs))):
        with pytest.raises(RuntimeError, match="autograd.Function"):
            transform()


def test_forward_and_backward_of_the_classes():
    import rwkv_cuda_b200 as R
    F = R.functions
    per_class = {"wkv4": F.WKV, "timex": F.TimeX, "wkv5": F.WKV_5, "wkv6": F.WKV_6, "wkv6 state": F.WKV_6STATE_EX,
                 "wkv7": F.RWKV7_CLAMPW_CUDA_OP, "wkv7 state": F.RWKV7_STATE_CLAMPW_CUDA_OP,
                 "wkv7 state passing": F.RWKV7_STATE_PASSING_CLAMPW_CUDA_OP}
    for name, cls in per_class.items():
        xs, call = cases()[name]
        xs = [x.cuda().requires_grad_(True) for x in xs]
        sub = type(cls.__name__ + "Sub", (cls,), {})
        lead = dict(wkv4=(2, 24, 32), wkv5=(2, 64, 128, 2), wkv6=(2, 64, 128, 2)).get(name, ())
        tail = (2, 8, 300, 0.1) if name == "timex" else ()
        a, b = call(*xs), sub.apply(*lead, *xs, *tail)
        assert outputs(b)[0].grad_fn.name() == sub.__name__ + "Backward" and outputs(a)[0].grad_fn.name() == cls.__name__ + "Backward"
        for p, q in zip(outputs(a), outputs(b)):
            assert torch.equal(p, q), name
        for p, q in zip(gradients(call, xs), gradients(lambda *x: sub.apply(*lead, *x, *tail), xs)):
            assert p.shape == q.shape and torch.equal(p, q), name


@pytest.mark.parametrize("name", NAMES)
def test_walks_unused_outputs_and_inputs_without_gradient(name):
    xs, call = cases()[name]
    xs = [x.cuda().requires_grad_(True) for x in xs]
    want = gradients(call, xs)
    ys = outputs(call(*xs))
    for a, b in zip(torch.autograd.grad(ys, xs, cotangents(ys), retain_graph=True), want):
        assert torch.equal(a, b)
    # an expanded gradient; an output that nothing depends on counts as one with a gradient of zero
    for y in ys:
        one = torch.autograd.grad(y, xs, torch.ones((), device="cuda", dtype=y.dtype).expand(y.shape), retain_graph=True)
        zero = [torch.ones_like(z) if z is y else torch.zeros_like(z) for z in ys]
        for a, b in zip(one, torch.autograd.grad(ys, xs, zero, retain_graph=True)):
            assert torch.equal(a, b)
    torch.autograd.grad(ys, xs, cotangents(ys))
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(ys, xs, cotangents(ys))
    some = [x.detach().requires_grad_(i % 2 == 0) for i, x in enumerate(xs)]
    got = gradients_of(call, some, some[::2])
    for a, b in zip(got, want[::2]):
        assert torch.equal(a, b)
    assert not outputs(call(*(x.detach() for x in xs)))[0].requires_grad
    with torch.no_grad():
        assert not outputs(call(*xs))[0].requires_grad


def gradients_of(call, xs, wanted):
    ys = outputs(call(*xs))
    return torch.autograd.grad(ys, wanted, cotangents(ys))


@pytest.mark.parametrize("name", NAMES)
def test_two_streams_and_two_threads(name):
    """The same call on two streams of two threads at once: every one gets the gradients of a call alone."""
    import threading
    xs, call = cases()[name]
    xs = [x.cuda() for x in xs]
    want = gradients(call, [x.clone().requires_grad_(True) for x in xs])
    torch.cuda.synchronize()
    wrong = []

    def work():
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                got = gradients(call, [x.clone().requires_grad_(True) for x in xs])
                torch.cuda.current_stream().synchronize()
                if not all(torch.equal(a, b) for a, b in zip(got, want)):
                    wrong.append(name)

    threads = [threading.Thread(target=work) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.parametrize("what", ["update", "training"])
def test_other_threads_run_while_a_launch_waits(what):
    """A launch waits when the GPU's queue is full (behind a kernel that takes half a second here); other Python threads go on."""
    import threading
    import time
    import rwkv_cuda_b200 as R
    if what == "training":
        xs, fn = cases()["wkv4"]
        xs = [x.cuda() for x in xs]
        call = lambda: fn(*xs)
    else:
        xs = [x.cuda() for x in cases()["wkv7 state"][0]]
        one = [x[:, :1].contiguous() for x in xs[1:]]
        y = torch.empty_like(one[0])
        call = lambda: R.ops.wkv7_state_update(xs[0], *one, y)
    call()
    torch.cuda.synchronize()
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0.001)

    thread = threading.Thread(target=tick)
    thread.start()
    t0 = time.perf_counter()
    torch.cuda._sleep(1_000_000_000)
    for _ in range(3000):
        call()
    waited = time.perf_counter() - t0
    stop.set()
    thread.join()
    torch.cuda.synchronize()
    assert waited > 0.25, "the queue never filled up"
    assert max(b - a for a, b in zip(ticks, ticks[1:])) < 0.5 * waited


@pytest.mark.parametrize("name", [n for n in NAMES if not n.startswith("wkv7")])   # (RWKV-7 refuses such tensors everywhere)
def test_gradients_that_are_not_aligned(name):
    """A contiguous gradient that starts anywhere in a larger one, as autograd hands it over when outputs are flattened and
    concatenated.  Every class computes it; the aligned call differs by rounding."""
    xs, call = cases()[name]
    xs = [x.cuda().requires_grad_(True) for x in xs]
    ys = outputs(call(*xs))
    flat = torch.cat([torch.zeros(1, device="cuda")] + [y.float().flatten() for y in ys])
    want = torch.autograd.grad(ys, xs, cotangents(ys), retain_graph=True)
    odd = []
    for c in cotangents(ys):
        whole = torch.empty(c.numel() + 1, dtype=c.dtype, device="cuda")
        whole[1:] = c.flatten()
        odd.append(whole[1:].view(c.shape))
        assert odd[-1].is_contiguous() and odd[-1].data_ptr() % 16
    tol = Hh.TOL_BF16 if any(x.dtype == BF for x in xs) else Hh.TOL_FP32
    for a, b in zip(torch.autograd.grad(ys, xs, odd, retain_graph=True), want):
        Hh.assert_close(a, b.double().cpu(), tol, name)
    whole = torch.autograd.grad(flat.square().sum(), xs, retain_graph=True)
    for a, b in zip(whole, torch.autograd.grad(ys, xs, [2 * y.detach() for y in ys])):
        Hh.assert_close(a, b.double().cpu(), tol, name)
