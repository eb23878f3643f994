"""The FP32 GEMM work that programs give this framework, through its public entry points.

Three entry points are covered: `flash_train.torch.gemm` (dense tensors), a Plan of the staged API that a program
makes once and executes on every step (strided views, the products of a Linear layer), and a Plan of the grouped
GEMM (the experts of a mixture-of-experts layer). Sizes are those of the repository's benchmark configurations and
test sweeps, and ragged ones around them.

Run from the repository root on a built tree.
"""
import math
import sys
from pathlib import Path

import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "flash-train_b200" / "python"))

import flash_train.torch as ft  # noqa: E402
from flash_train import capi  # noqa: E402

# How a case reaches the library ("via"):
#   torch    flash_train.torch.gemm(a, b, c, alpha, beta), everything dense row-major
#   plan     a Plan of the staged API, executed with the workspace it asks for; "a_t" / "b_t": the operand is the
#            transposed view of a dense buffer
#   grouped  a Plan of GroupedABCDGemm over "groups" groups of different row counts (one of them empty)


def listed():
    return [
        # A tiny dense product (the first benchmark configuration): nothing but latency and launches.
        {"name": "tiny_128x64x96", "via": "torch", "m": 128, "k": 64, "n": 96},
        # One token through the up-projection of an 8B-class MLP: the weight is streamed once.
        {"name": "decode_1x4096x14336", "via": "torch", "m": 1, "k": 4096, "n": 14336},
        # A decode batch of 32 through a square projection.
        {"name": "decode_32x4096x4096", "via": "torch", "m": 32, "k": 4096, "n": 4096},
        # A short ragged prompt (tail sweep of the benchmark configurations).
        {"name": "prompt_255x4096x4096", "via": "torch", "m": 255, "k": 4096, "n": 4096},
        # A Plan made once and executed on every step (Plan-reuse configuration).
        {"name": "plan_1024x1024x1024", "via": "plan", "m": 1024, "k": 1024, "n": 1024},
        # Forward pass of a Linear layer, y = x W^T: the weight is a transposed view.
        {"name": "linear_fwd_2048x4096x3072", "via": "plan", "m": 2048, "k": 4096, "n": 3072, "b_t": True},
        # Its weight gradient, dW = dy^T x: the gradient is a transposed view, the depth is the token count.
        {"name": "linear_wgrad_3072x8192x2048", "via": "plan", "m": 3072, "k": 8192, "n": 2048, "a_t": True},
        # alpha A B + beta C (addend configuration).
        {"name": "addend_4096x4096x4096", "via": "torch", "m": 4096, "k": 4096, "n": 4096, "c": True},
        # The transposed view of a buffer with an odd pitch (tail sweep).
        {"name": "ragged_4097x4096x4096_at", "via": "plan", "m": 4097, "k": 4096, "n": 4096, "a_t": True, "dist": "uniform"},
        # Eight experts with ragged token counts, one without tokens.
        {"name": "grouped_8192x4096x4096", "via": "grouped", "m": 8192, "k": 4096, "n": 4096, "groups": 8},
        # Training: up-projection of an 8B-class MLP over 16384 tokens (the headline configuration).
        {"name": "train_16384x4096x14336", "via": "torch", "m": 16384, "k": 4096, "n": 14336, "dist": "weights"},
        # A small output with a very deep sum (tall-K configuration).
        {"name": "tall_2048x262144x2048", "via": "torch", "m": 2048, "k": 262144, "n": 2048, "dist": "uniform"},
    ]


def _spread(rng, low, high, odd=0.35):
    """A size between low and high, even over the logarithm; a multiple of 64 / 8 / 1 by chance."""
    size = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    if rng.random() > odd:
        unit = 64 if size >= 512 else 8
        size = max(unit, size // unit * unit)
    return min(max(size, low), high)


def draw(rng):
    kind = rng.choice(["tiny", "decode", "batch", "prompt", "middle", "linear", "wgrad", "train", "tall", "grouped"])
    case = {"via": "torch"}
    if kind == "tiny":
        case.update(m=_spread(rng, 33, 320), k=_spread(rng, 32, 512), n=_spread(rng, 32, 320))
    elif kind == "decode":
        case.update(m=rng.randint(1, 8), k=_spread(rng, 1024, 14336, 0), n=_spread(rng, 1024, 14336, 0))
    elif kind == "batch":
        case.update(m=rng.randint(9, 64), k=_spread(rng, 1024, 8192, 0.1), n=_spread(rng, 1024, 14336, 0.1))
    elif kind == "prompt":
        case.update(m=_spread(rng, 65, 512), k=_spread(rng, 1024, 8192, 0.1), n=_spread(rng, 1024, 14336, 0.1))
    elif kind == "middle":
        case.update(via="plan", m=_spread(rng, 384, 2048), k=_spread(rng, 512, 4096), n=_spread(rng, 384, 2048))
    elif kind == "linear":
        case.update(via="plan", m=_spread(rng, 512, 8192), k=_spread(rng, 512, 8192, 0.1), n=_spread(rng, 512, 8192, 0.1), b_t=True)
    elif kind == "wgrad":
        case.update(via="plan", m=_spread(rng, 512, 8192, 0.1), k=_spread(rng, 1024, 16384), n=_spread(rng, 512, 4096, 0.1), a_t=True)
    elif kind == "train":
        case.update(m=_spread(rng, 2048, 16384), k=_spread(rng, 1024, 4096, 0.1), n=_spread(rng, 1024, 14336, 0.1), dist="weights")
    elif kind == "tall":
        case.update(m=_spread(rng, 256, 2048, 0.1), k=_spread(rng, 16384, 262144, 0.1), n=_spread(rng, 256, 2048, 0.1), dist="uniform")
    else:
        case.update(via="grouped", m=_spread(rng, 1024, 16384), k=_spread(rng, 512, 4096, 0) // 8 * 8,
                    n=_spread(rng, 512, 4096, 0) // 8 * 8, groups=rng.randint(2, 16))
    if case["via"] != "grouped" and rng.random() < 0.25:
        case["c"] = True
    return case


def _group_rows(case):
    """Ragged row counts that sum to m; the second group has none."""
    groups, m = case["groups"], case["m"]
    weights = [0 if g == 1 else 1 + (7 * g + 3) % 5 for g in range(groups)]
    rows = [m * w // sum(weights) for w in weights]
    rows[0] += m - sum(rows)
    return rows


def _matrix(rows, cols, dist, scale, generator):
    if dist == "uniform":
        return torch.rand(rows, cols, device="cuda", generator=generator).mul_(2).sub_(1)
    return torch.randn(rows, cols, device="cuda", generator=generator).mul_(scale)


def _inputs(case, seed):
    """a, b, c, alpha, beta; for a grouped case a and b hold the groups' matrices one below the other."""
    generator = torch.Generator(device="cuda").manual_seed(seed)
    m, k, n = case["m"], case["k"], case["n"]
    dist = case.get("dist", "normal")
    weight = k ** -0.5 if dist == "weights" else 1.0
    depth = k * case["groups"] if case["via"] == "grouped" else k
    a = _matrix(k, m, dist, 1.0, generator).t() if case.get("a_t") else _matrix(m, k, dist, 1.0, generator)
    b = _matrix(n, k, dist, weight, generator).t() if case.get("b_t") else _matrix(depth, n, dist, weight, generator)
    c = _matrix(m, n, dist, 1.0, generator) if case.get("c") else None
    return a, b, c, (1.5 if c is not None else 1.0), (0.5 if c is not None else 0.0)


def prepare(case, seed):
    a, b, c, alpha, beta = _inputs(case, seed)
    m, k, n = case["m"], case["k"], case["n"]
    state = {"via": case["via"], "a": a, "b": b, "c": c, "alpha": alpha, "beta": beta}
    if case["via"] == "torch":
        return state
    state["d"] = torch.empty(m, n, device="cuda")
    if case["via"] == "plan":
        c_operand = capi.null_operand(m, n) if c is None else capi.tensor_operand(c)
        state["plan"] = capi.GemmBinding().make_plan(capi.tensor_operand(a), capi.tensor_operand(b), c_operand,
                                                     capi.tensor_operand(state["d"]), alpha, beta)
    else:
        rows, groups = _group_rows(case), case["groups"]
        state["plan"] = capi.GroupedGemmBinding().make_plan(
            {"address": a.data_ptr(), "rows": rows, "cols": [k] * groups},
            {"address": b.data_ptr(), "rows": [k] * groups, "cols": [n] * groups},
            {"address": 0, "rows": rows, "cols": [n] * groups},
            {"address": state["d"].data_ptr(), "rows": rows, "cols": [n] * groups}, alpha, beta)
    state["bytes"] = state["plan"].workspace_bytes(0)
    state["workspace"] = torch.empty(max(state["bytes"], 1), dtype=torch.uint8, device="cuda")
    return state


def run(state):
    if state["via"] == "torch":
        return ft.gemm(state["a"], state["b"], state["c"], state["alpha"], state["beta"])
    size = state["bytes"]
    state["plan"].execute(0, state["workspace"].data_ptr() if size else 0, size, torch.cuda.current_stream().cuda_stream)
    return state["d"]


def work(case):
    m, k, n = case["m"], case["k"], case["n"]
    weights = k * n
    if case["via"] == "grouped":
        weights *= sum(1 for rows in _group_rows(case) if rows)
    return {"bytes": 4.0 * (m * k + weights + m * n * (2 if case.get("c") else 1)), "flops": 2.0 * m * k * n}


def tolerance(case):
    # FP32 operands and FP32 sums: the error of a sum of k products grows like sqrt(k). Against float64 the path shows
    # 1.4e-7 at k = 64, 1.1e-6 at 4096 and 3.6e-6 at 262144 (slices summed apart); a strictly sequential FP32 sum
    # is at about 0.3 * 2^-24 sqrt(k). About four times that.
    return {"rel": 2.0 ** -24 * max(10.0, math.sqrt(case["k"]))}


def exact(case, seed):
    a, b, c, alpha, beta = _inputs(case, seed)
    m, k, n = case["m"], case["k"], case["n"]
    d = torch.zeros(m, n, dtype=torch.float64, device="cuda")
    if case["via"] == "grouped":
        first = 0
        for g, rows in enumerate(_group_rows(case)):
            d[first:first + rows] = a[first:first + rows].double() @ b[g * k:(g + 1) * k].double()
            first += rows
        return d
    for at in range(0, k, 16384):
        d += a[:, at:at + 16384].double() @ b[at:at + 16384].double()
    d *= alpha
    return d if c is None else d + beta * c.double()
