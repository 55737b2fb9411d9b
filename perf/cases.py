"""Performance cases of the operators: the calls that training and inference programs make, over the sizes they make
them at.

A case names an operator family ("op"), the activation type and the sizes:

  wkv7_update   RWKV-7 inference, `ops.wkv7_state_update`: T = 1 is a decoding step, a longer T a prompt (of any length)
  wkv7          RWKV-7 training step with state passing (forward + backward), T a multiple of 16 as the operator asks
  wkv6state     RWKV-6 training step with fp32 state in and out
  wkv6          RWKV-6 training step without a state, any T
  wkv5          RWKV-5 training step, bf16 or fp32
  wkv4          RWKV-4 training step, fp32
  timex         depthwise_conv1d training step, fp32

Head size is 64 throughout, the size that RWKV models use.  Inputs follow the distributions of the benchmark
configurations.  A training step is what autograd runs: `apply`, then the gradients of every input.
"""
import math

import torch

import rwkv_cuda_b200 as R

N = 64
BF16, F32 = "bf16", "f32"


def listed():
    return [
        # one sequence being decoded on a small model (12 heads): launch latency is all there is
        dict(name="rwkv7 decode B1", op="wkv7_update", dtype=BF16, B=1, T=1, H=12),
        # a decoding step of a serving batch: the states (128 x 32 x 16 KB) are read and written once
        dict(name="rwkv7 decode B128", op="wkv7_update", dtype=BF16, B=128, T=1, H=32),
        # one prompt of a length that nobody padded
        dict(name="rwkv7 prompt T1999", op="wkv7_update", dtype=BF16, B=1, T=1999, H=32),
        # fine-tuning a small model on short sequences; T is 32.5 chunks of 32 tokens
        dict(name="rwkv7 train small", op="wkv7", dtype=BF16, B=2, T=1040, H=12),
        # the benchmark configuration of RWKV-7
        dict(name="rwkv7 train B16 T4096", op="wkv7", dtype=BF16, B=16, T=4096, H=64),
        # the benchmark configuration of RWKV-6 with state
        dict(name="rwkv6 state train B16 T4096", op="wkv6state", dtype=BF16, B=16, T=4096, H=64),
        # RWKV-6 on documents cut at 1000 tokens
        dict(name="rwkv6 train T1000", op="wkv6", dtype=BF16, B=8, T=1000, H=32),
        # the benchmark configuration of RWKV-5
        dict(name="rwkv5 train B8 T4096", op="wkv5", dtype=BF16, B=8, T=4096, H=64),
        # RWKV-5 trained in fp32, as the reference's fp32 harness does
        dict(name="rwkv5 train fp32", op="wkv5", dtype=F32, B=8, T=512, H=16),
        # the benchmark configuration of RWKV-4
        dict(name="rwkv4 train B4 T256", op="wkv4", dtype=F32, B=4, T=256, C=256),
        # an ordinary RWKV-4 training batch
        dict(name="rwkv4 train B32 T768", op="wkv4", dtype=F32, B=32, T=768, C=768),
        # the benchmark configuration of depthwise_conv1d
        dict(name="conv1d train B32 T768", op="timex", dtype=F32, B=32, T=768, C=768),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    op = rng.choice(["decode", "prompt", "wkv7", "wkv6state", "wkv6", "wkv5", "wkv5 fp32", "wkv4", "timex"])
    if op in ("wkv4", "timex"):
        while True:
            c = dict(op=op, dtype=F32, B=_log_int(rng, 1, 32), T=_log_int(rng, 32, 1024), C=_log_int(rng, 64, 1024))
            if op == "wkv4" or c["B"] * c["C"] * c["T"] ** 2 <= 32 * 768 * 768 ** 2:
                return c
    H = rng.choice([8, 12, 16, 24, 32, 40, 64])
    if op == "decode":      # serving batches
        return dict(op="wkv7_update", dtype=BF16, B=_log_int(rng, 1, 256), T=1, H=H)
    if op == "prompt":
        return dict(op="wkv7_update", dtype=BF16, B=_log_int(rng, 1, 4), T=_log_int(rng, 16, 4096), H=H)
    if op == "wkv5 fp32":
        return dict(op="wkv5", dtype=F32, B=_log_int(rng, 1, 8), T=_log_int(rng, 64, 512), H=rng.choice([8, 12, 16]))
    B, T = _log_int(rng, 1, 16), _log_int(rng, 128, 4096)
    if op in ("wkv5", "wkv6") and rng.random() < 0.5:   # sequences of any length, shorter ones
        return dict(op=op, dtype=BF16, B=min(B, 8), T=min(T, 1024), H=min(H, 32))
    return dict(op=op, dtype=BF16, B=min(B, 8) if op == "wkv5" else B, T=(T + 15) // 16 * 16, H=H)


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    op, B, T = case["op"], case["B"], case["T"]
    dt = torch.bfloat16 if case["dtype"] == BF16 else torch.float32
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    ru = lambda lo, hi, *s: torch.rand(*s, device="cuda", generator=g) * (hi - lo) + lo
    st = dict(case)
    if op == "wkv4":
        C = case["C"]
        st["in"] = [ru(-4, 1, C), ru(-1, 1, C), 0.5 * rn(B, T, C), rn(B, T, C)]
        st["g"] = [rn(B, T, C)]
    elif op == "timex":
        C = case["C"]
        st["in"] = [rn(C, T) / T ** 0.5, rn(B, C, T)]
        st["g"] = [rn(B, C, T)]
    elif op in ("wkv7", "wkv7_update"):
        H = case["H"]
        r, k, v = ((0.5 * rn(B, T, H, N)).to(dt) for _ in range(3))
        w = rn(B, T, H, N).to(dt)
        kk = torch.nn.functional.normalize(rn(B, T, H, N), dim=-1)
        a, b = (-kk).to(dt), (kk * torch.sigmoid(rn(B, T, H, N))).to(dt)
        st["in"] = [0.1 * rn(B, H, N, N), r, w, k, v, a, b]
        if op == "wkv7":
            st["g"] = [rn(B, T, H * N).to(dt), rn(B, H, N, N)]
    else:
        H = case["H"]
        C = H * N
        r, k, v = ((0.5 * rn(B, T, C)).to(dt) for _ in range(3))
        u = ru(-1, 1, H, N).to(dt)
        w = ru(-6, -1, H, N).to(dt) if op == "wkv5" else (rn(B, T, C) - 5.0).to(dt)
        st["in"], st["g"] = [r, k, v, w, u], [rn(B, T, C).to(dt)]
        if op == "wkv6state":
            st["in"].append(0.1 * rn(B, H, N, N))
            st["g"].append(rn(B, H, N, N))
    if op != "wkv7_update":
        for x in st["in"]:
            x.requires_grad_(True)
    return st


def run(st):
    op, B, T, F = st["op"], st["B"], st["T"], R.functions
    if op == "wkv7_update":
        y = torch.empty_like(st["in"][1])
        R.ops.wkv7_state_update(*st["in"], y)
        return y, st["in"][0]
    if op == "wkv7":
        out = F.RWKV7_STATE_PASSING_CLAMPW_CUDA_OP.apply(*st["in"])
    elif op == "wkv6state":
        out = F.WKV_6STATE_EX.apply(*st["in"])
    elif op == "wkv6":
        out = F.WKV_6.apply(B, T, st["H"] * N, st["H"], *st["in"])
    elif op == "wkv5":
        out = F.WKV_5.apply(B, T, st["H"] * N, st["H"], *st["in"])
    elif op == "wkv4":
        out = F.WKV.apply(B, T, st["C"], *st["in"])
    else:
        out = F.TimeX.apply(*st["in"], B, st["C"], T, 0.1)
    out = out if isinstance(out, tuple) else (out,)
    return out, torch.autograd.grad(out, st["in"], st["g"])


def work(case):
    """Bytes: every input read once and every output written once, forward and backward each (the backward reads the
    forward's inputs again).  Operations: those of the recurrence, token by token, per state element; for the
    convolution its three correlations."""
    op, B, T = case["op"], case["B"], case["T"]
    e = 2 if case["dtype"] == BF16 else 4
    if op == "wkv4":
        n = B * T * case["C"]
        return dict(bytes=32 * n + 16 * case["C"], flops=40 * n)
    if op == "timex":
        C = case["C"]
        return dict(bytes=4 * (5 * B * C * T + 3 * C * T), flops=3 * B * C * T * (T + 1))
    H = case["H"]
    n, states = B * T * H * N, 4 * B * H * N * N
    if op == "wkv7_update":
        return dict(bytes=7 * e * n + 2 * states, flops=9 * n * N)
    fwd, bwd, st, fl = {"wkv7": (7, 13, 4, 31), "wkv6state": (5, 9, 4, 19), "wkv6": (5, 9, 0, 19), "wkv5": (4, 7, 0, 19)}[op]
    return dict(bytes=(fwd + bwd) * e * n + st * states, flops=fl * n * N)


def tolerance(case):
    if case["dtype"] == BF16:
        return dict(rel=1e-2, max=0.15)
    # fp32 sums over at most 32 x 1024 tokens; the RWKV-5 decay gradient weights its terms by their distance in time
    return dict(rel=1e-5 if case["op"] == "timex" else 2e-5)
