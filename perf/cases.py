"""The work this library is measured on: log-space contractions through its public entry points.

A case is one call of `lm2exp` (out[r,i,k] = log sum_j a[r,i,j] exp b[r,j,k]) or `lt2exp` (out[r,s,k] = log sum_ij
w[r,s,i,j] exp a[r,i,k] exp b[r,j,k]) on operands that are resident on the GPU, as one layer of a circuit makes it.
Sizes are those of the five benchmark configurations (`triturus_b200/workloads.py`), of the reference's benchmark
sweeps (`triturus_b200/sweeps.py`) and of its tests (odd sizes).  `precision` is "3xtf32", the default of the library,
or "tf32", what `set_tf32_enabled(True)` selects.
"""

import math

import torch

import triturus_b200 as tb

NEG_INF = float("-inf")


def listed():
    return [
        # One small layer of a single circuit, nothing batched: launch and host latency count.
        {"name": "lm2exp 1x128^3 3x", "op": "lm2exp", "precision": "3xtf32", "dist": "normal", "R": 1, "I": 128, "J": 128, "K": 128},
        # A few small dense layers with normalised weights over log-probabilities.
        {"name": "lm2exp 4x256^3", "op": "lm2exp", "precision": "tf32", "dist": "softmax", "R": 4, "I": 256, "J": 256, "K": 256},
        # Layer widths and a data batch that are no multiple of anything (rows not 16-byte aligned).
        {"name": "lm2exp 24x150x101x203 3x", "op": "lm2exp", "precision": "3xtf32", "dist": "normal", "R": 24, "I": 150, "J": 101, "K": 203},
        # A batch of medium layers over a data batch of 256, default precision.
        {"name": "lm2exp 64x512x512x256 3x", "op": "lm2exp", "precision": "3xtf32", "dist": "normal", "R": 64, "I": 512, "J": 512, "K": 256},
        # Wide layers, columns at very different levels and with impossible states (-inf): bound by the tensor cores.
        {"name": "lm2exp 32x1024^3", "op": "lm2exp", "precision": "tf32", "dist": "offset", "R": 32, "I": 1024, "J": 1024, "K": 1024},
        # The same at the default precision.
        {"name": "lm2exp 32x1024^3 3x", "op": "lm2exp", "precision": "3xtf32", "dist": "offset", "R": 32, "I": 1024, "J": 1024, "K": 1024},
        # Many narrow layers over a large data batch: bound by memory.
        {"name": "lm2exp 128x256x256x8192", "op": "lm2exp", "precision": "tf32", "dist": "softmax", "R": 128, "I": 256, "J": 256, "K": 8192},
        # A small bilinear (Tucker) layer of odd widths.
        {"name": "lt2exp 3x75x50x50x100 3x", "op": "lt2exp", "precision": "3xtf32", "dist": "normal", "R": 3, "S": 75, "I": 50, "J": 50, "K": 100},
        # One bilinear layer of a single circuit: few output tiles, a long contraction.
        {"name": "lt2exp 1x256^4 3x", "op": "lt2exp", "precision": "3xtf32", "dist": "normal", "R": 1, "S": 256, "I": 256, "J": 256, "K": 256},
        # A batch of bilinear layers of moderate width.
        {"name": "lt2exp 16x128x64x64x2048", "op": "lt2exp", "precision": "tf32", "dist": "softmax", "R": 16, "S": 128, "I": 64, "J": 64, "K": 2048},
        # Wide bilinear layers over a large data batch, with impossible states: the longest call.
        {"name": "lt2exp 64x256x128x128x4096", "op": "lt2exp", "precision": "tf32", "dist": "offset", "R": 64, "S": 256, "I": 128, "J": 128, "K": 4096},
        # Wide bilinear layers over a data batch of 256, default precision: the weights are most of the bytes.
        {"name": "lt2exp 32x256^4 3x", "op": "lt2exp", "precision": "3xtf32", "dist": "normal", "R": 32, "S": 256, "I": 256, "J": 256, "K": 256},
    ]  # fmt: skip


def _size(rng, low, high):
    """A size of the range, spread over its logarithm: half of them round (multiples of 32), half as they come."""
    x = math.exp(rng.uniform(math.log(low), math.log(high)))
    if rng.random() < 0.5:
        return max(low, min(high, 32 * round(x / 32)))
    return max(low, min(high, round(x)))


def draw(rng):
    """One more case: layers of 64 ... 1024 units (lm2exp) or 32 ... 256 (lt2exp), 1 ... 128 layers, 64 ... 8192 columns."""
    while True:
        case = {"op": rng.choice(["lm2exp", "lt2exp"]), "precision": rng.choice(["tf32", "3xtf32"]), "dist": rng.choice(["normal", "softmax", "offset"])}
        if case["op"] == "lm2exp":
            case.update(R=max(1, round(math.exp(rng.uniform(0, math.log(128))))), I=_size(rng, 64, 1024), J=_size(rng, 64, 1024), K=_size(rng, 64, 8192))
        else:
            case.update(R=max(1, round(math.exp(rng.uniform(0, math.log(64))))), S=_size(rng, 32, 256), I=_size(rng, 32, 256), J=_size(rng, 32, 256), K=_size(rng, 64, 4096))
        w = work(case)
        # no more time than the largest listed case takes: three tensor-core products per term at the default precision
        if w["bytes"] <= 2.2e9 and w["flops"] <= (2.1e12 if case["precision"] == "tf32" else 3.5e11):
            return case


def _log_values(g, R, N, K, dist):
    """Log-space values [R, N, K]: what the layer below hands up."""
    x = torch.randn(R, N, K, generator=g, device="cuda")
    if dist == "softmax":  # log-probabilities over the units of a layer, each column at a level of its own
        return torch.log_softmax(3.0 * x, dim=1) - 50.0 * torch.rand(R, 1, K, generator=g, device="cuda")
    if dist == "offset":  # far-apart levels and impossible states
        x = -20.0 + 10.0 * x + (400.0 * torch.rand(R, 1, K, generator=g, device="cuda") - 200.0)
        return x.masked_fill_(torch.rand(R, N, K, generator=g, device="cuda") < 0.01, NEG_INF)
    return x


def prepare(case, seed):
    """The weights and the log-space operands on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    R, I, J, K, dist = case["R"], case["I"], case["J"], case["K"], case["dist"]
    S = case.get("S")
    shape = (R, I, J) if S is None else (R, S, I * J)
    if dist == "softmax":
        w = torch.softmax(torch.randn(*shape, generator=g, device="cuda"), dim=-1)
    else:
        w = torch.rand(*shape, generator=g, device="cuda")
        if dist == "offset":  # weights that sum to one
            w /= w.sum(-1, keepdim=True)
    if S is None:
        operands = (w, _log_values(g, R, J, K, dist))
    else:
        operands = (w.view(R, S, I, J), _log_values(g, R, I, K, dist), _log_values(g, R, J, K, dist))
    return {"op": tb.lm2exp if S is None else tb.lt2exp, "operands": operands, "precision": case["precision"]}


def run(state):
    return state["op"](*state["operands"], precision=state["precision"])


def work(case):
    """Operands read once, result written once, in 32-bit floats; two operations per term of the contraction."""
    R, I, J, K = case["R"], case["I"], case["J"], case["K"]
    if case["op"] == "lm2exp":
        return {"bytes": 4 * R * (I * J + J * K + I * K), "flops": 2 * R * I * J * K}
    S = case["S"]
    return {"bytes": 4 * R * (S * I * J + I * K + J * K + S * K), "flops": 2 * R * S * I * J * K}


def tolerance(case):
    """Four times the distance from the same contraction in 64 bits, measured over the listed cases and a dozen others.

    tf32: operands of 11 significant bits, log-space errors up to 1.4e-3 (rel 1.1e-5, max 4.1e-5 where the columns lie
    far from zero; rel 8.4e-5, max 1.4e-4 where the results are 4 ... 10).  3xtf32: rel 1.4e-6, max 1.9e-6."""
    if case["precision"] == "3xtf32":
        return {"rel": 6e-6, "max": 8e-6}
    return {"rel": 3.4e-4, "max": 5.6e-4} if case["dist"] == "normal" else {"rel": 5e-5, "max": 2e-4}
