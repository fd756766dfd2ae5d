"""The calls a program makes of this library, as timed cases.

Each case is one call (or one training step) through the Python entry points
on operands that are already on the GPU: the plain product over its range of
sizes and layouts, the Gram product, block orthogonalisation, a training step
through autograd, the split-precision product and a batch of products.
"""
import math
import random

import torch

import tsm_benchmark_b200 as tsm
from tsm_benchmark_b200 import autograd, batched

DTYPES = {"f64": torch.float64, "f32": torch.float32}

# The most a drawn case may ask for: bytes in and out, and multiply-adds x 2.
MAX_BYTES = 2.0e9
MAX_FLOPS = 1.7e10


def listed():
    return [
        # The shortest call: a projection inside an iteration on a small
        # problem (8 vectors, 4096 rows), where latency counts.
        {"name": "small-8x8", "op": "plain", "dtype": "f64", "layout": "rows", "n": 4096, "m": 8, "k": 8},
        # The reference driver's row count with its widest default block.
        {"name": "driver-16x16", "op": "plain", "dtype": "f64", "layout": "rows", "n": 1 << 20, "m": 16, "k": 16},
        # The benchmark's headline shape.
        {"name": "headline-8x8", "op": "plain", "dtype": "f64", "layout": "rows", "n": 1 << 26, "m": 8, "k": 8},
        # A block eigensolver's 24 vectors on a grid of a few million points.
        {"name": "even-24x24", "op": "plain", "dtype": "f64", "layout": "rows", "n": 2000003, "m": 24, "k": 24},
        # A basis that has grown to 37 vectors against 13 new ones.
        {"name": "odd-37x13", "op": "plain", "dtype": "f64", "layout": "rows", "n": 700001, "m": 37, "k": 13},
        # The widest products, bound by arithmetic.
        {"name": "wide-64x64", "op": "plain", "dtype": "f64", "layout": "rows", "n": 1 << 21, "m": 64, "k": 64},
        # A Krylov basis kept in one row-major matrix: its leading 40 columns
        # against the 20 after them, both read in place.
        {"name": "slices-40x20", "op": "plain", "dtype": "f64", "layout": "slice", "n": 1 << 20, "m": 40, "k": 20},
        # The Gram matrix of 32 vectors (Cholesky QR).
        {"name": "gram-32", "op": "gram", "dtype": "f64", "layout": "rows", "n": 1 << 22, "m": 32, "k": 32},
        # One block Gram-Schmidt step: 8 new vectors against a basis of 32.
        {"name": "orth-32x8", "op": "orth", "dtype": "f64", "layout": "rows", "n": 1 << 20, "m": 32, "k": 8},
        # A training step through the product: forward, loss, both gradients.
        {"name": "train-f32-16x16", "op": "train", "dtype": "f32", "layout": "rows", "n": 1 << 22, "m": 16, "k": 16},
        # FP32 data at the precision the FP32 kernels do not reach.
        {"name": "split-32x32", "op": "split", "dtype": "f32", "layout": "rows", "n": 1 << 24, "m": 32, "k": 32,
         "kind": "tf32"},
        # Many products of uneven rows and widths in one launch.
        {"name": "batch-128", "op": "batch", "dtype": "f64", "count": 128, "nmin": 1000, "nmax": 1000000, "mix": 1},
    ]


def _logint(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(["plain"] * 5 + ["gram", "orth", "train", "split", "batch"])
    if op == "batch":
        case = {"op": op, "dtype": "f64", "count": _logint(rng, 8, 200), "nmin": 1000,
                "nmax": _logint(rng, 10000, 1000000), "mix": rng.randrange(1 << 30)}
        while work(case)["bytes"] > MAX_BYTES or work(case)["flops"] > MAX_FLOPS:
            case["count"] = max(1, case["count"] // 2)
        return case
    dtype = "f64" if op in ("gram", "orth") else "f32" if op == "split" else rng.choice(["f64", "f64", "f32"])
    wide = 32 if op == "split" else 64
    case = {"op": op, "dtype": dtype, "layout": "rows", "n": _logint(rng, 1000, 1 << 26),
            "m": _logint(rng, 1, wide), "k": _logint(rng, 1, wide)}
    if op == "gram":
        case["k"] = case["m"]
    if op == "split":
        case["kind"] = rng.choice(["tf32", "tf32", "bf16x3", "bf16x2"])
        if case["kind"] != "tf32":
            case["m"], case["k"] = -(-case["m"] // 4) * 4, -(-case["k"] // 4) * 4
    if op == "plain":
        layouts = ["rows"] * 4 + ["slice"] * 2 + (["cols"] * 2 + ["mixed"] if dtype == "f64" else [])
        case["layout"] = rng.choice(layouts)
    while work(case)["bytes"] > MAX_BYTES or work(case)["flops"] > MAX_FLOPS:
        case["n"] = max(1000, int(case["n"] * rng.uniform(0.3, 0.9)))
    return case


def _problems(case):
    """(n, m, k) of every product of a batch."""
    rng = random.Random(case["mix"])
    return [(_logint(rng, case["nmin"], case["nmax"]), rng.choice((4, 8, 16, 32)), rng.choice((4, 8, 16, 32)))
            for _ in range(case["count"])]


def work(case):
    if case["op"] == "batch":
        probs = _problems(case)
        return {"bytes": 8.0 * sum(n * (m + k) + m * k for n, m, k in probs),
                "flops": 2.0 * sum(n * m * k for n, m, k in probs)}
    n, m, k = float(case["n"]), case["m"], case["k"]
    e = 8.0 if case["dtype"] == "f64" else 4.0
    if case["op"] == "gram":  # A in, C out; the upper triangle's products
        return {"bytes": e * (n * m + m * m), "flops": n * m * (m + 1)}
    if case["op"] == "orth":  # A and B in, B and C out
        return {"bytes": e * (n * (m + 2 * k) + m * k), "flops": 4.0 * n * m * k}
    if case["op"] == "train":  # A, B and W in; C, dA and dB out
        return {"bytes": e * (2 * n * (m + k) + 2 * m * k), "flops": 6.0 * n * m * k}
    out = 8.0 if case["op"] == "split" else e
    return {"bytes": e * n * (m + k) + out * m * k, "flops": 2.0 * n * m * k}


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _inputs(case, seed):
    """The operands: entries uniform in [-1, 1), as the reference's drivers
    have them; normal with columns of uneven scale for the split product."""
    g = _generator(seed)
    dt = DTYPES[case["dtype"]]

    def uniform(*shape):
        return torch.empty(shape, dtype=dt, device="cuda").uniform_(-1.0, 1.0, generator=g)

    if case["op"] == "batch":
        return [(uniform(n, m), uniform(n, k)) for n, m, k in _problems(case)]
    n, m, k = case["n"], case["m"], case["k"]
    if case["op"] == "split":
        def scaled(w):
            x = torch.empty((n, w), dtype=dt, device="cuda").normal_(generator=g)
            return x.mul_(10.0 ** torch.empty(w, device="cuda").uniform_(-3.0, 3.0, generator=g))
        return scaled(m), scaled(k)
    if case["layout"] == "slice":  # two neighbouring column blocks of one basis
        V = uniform(n, m + k)
        return V[:, :m], V[:, m:]
    A = uniform(m, n).t() if case["layout"] == "cols" else uniform(n, m)
    if case["op"] == "gram":
        return A, A
    if case["op"] == "orth":
        # Columns of norm sqrt(2): B - A (A^T B) is then a block reflection,
        # which can be applied to its own result again and again.
        A = A * math.sqrt(6.0 / n)
        if m <= n:
            L = torch.linalg.cholesky(A.t() @ A)
            A = (math.sqrt(2.0) * torch.linalg.solve_triangular(L, A.t().contiguous(), upper=False)).t().contiguous()
    B = uniform(k, n).t() if case["layout"] in ("cols", "mixed") else uniform(n, k)
    return A, B


def prepare(case, seed):
    x = _inputs(case, seed)
    state = {"op": case["op"], "x": x}
    if case["op"] == "batch":
        sizes = [a.shape[1] * b.shape[1] for a, b in x]
        flat = torch.zeros(sum(sizes), dtype=torch.float64, device="cuda")
        outs = [c.view(a.shape[1], b.shape[1]) for c, (a, b) in zip(flat.split(sizes), x)]
        state["flat"] = flat
        state["plan"] = batched.BatchedTSMTTSM([a for a, _ in x], [b for _, b in x], outs)
    elif case["op"] == "train":
        A, B = x
        state["x"] = (A.requires_grad_(), B.requires_grad_())
        state["W"] = torch.empty((case["m"], case["k"]), dtype=A.dtype, device="cuda").normal_(
            generator=_generator(seed + 1000003))
    elif case["op"] == "split":
        state["kind"] = case["kind"]
    return state


def run(state):
    op = state["op"]
    if op == "batch":
        state["plan"].run()
        return state["flat"]
    A, B = state["x"]
    if op == "plain":
        return tsm.tsmttsm(A, B)
    if op == "gram":
        return tsm.gram(A)
    if op == "orth":
        C = tsm.block_orthogonalize(A, B)
        return C, B
    if op == "split":
        return tsm.tsmttsm_split(A, B, kind=state["kind"])
    C = autograd.gram_tn(A, B)
    dA, dB = torch.autograd.grad((state["W"] * C).sum(), (A, B))
    return C.detach(), dA, dB


def _product(A, B):
    """A^T B in 64 bits, over blocks of rows."""
    C = torch.zeros((A.shape[1], B.shape[1]), dtype=torch.float64, device=A.device)
    step = 1 << 20
    for r in range(0, A.shape[0], step):
        C += A[r:r + step].double().t() @ B[r:r + step].double()
    return C


def exact(case, seed):
    x = _inputs(case, seed)
    if case["op"] == "batch":
        return torch.cat([_product(a, b).reshape(-1) for a, b in x])
    A, B = x
    C = _product(A, B)
    if case["op"] == "orth":
        return C, B - A @ C
    if case["op"] == "train":
        W = torch.empty((case["m"], case["k"]), dtype=A.dtype, device="cuda").normal_(
            generator=_generator(seed + 1000003)).double()
        return C, B.double() @ W.t(), A.double() @ W
    return C
