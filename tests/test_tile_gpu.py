"""The any-layout tensor-core kernel: every way an operand can lie in memory,
at the edges of tiles, chunks, phases and boxes, through the calls that reach
it, against A^T B in FP64.

FP64: the normwise bound 4 sqrt(n) 2^-53 ||A||_F ||B||_F.  FP32 storage is
multiplied and summed in FP64 and rounded once: half an ulp (2^-24) of each
entry on top of that bound.
"""
import itertools
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# layout -> operand of n x w
LAYOUTS = {
    "rows": lambda n, w, dt, dev: torch.randn(n, w, dtype=dt, device=dev),
    "even pitch": lambda n, w, dt, dev: torch.randn(n, w + 4 + w % 2, dtype=dt, device=dev)[:, :w],
    "odd pitch": lambda n, w, dt, dev: torch.randn(n, w + 3 + w % 2, dtype=dt, device=dev)[:, 1:w + 1],
    "unaligned": lambda n, w, dt, dev: torch.randn(n * w + 1, dtype=dt, device=dev)[1:].view(n, w),
    "columns": lambda n, w, dt, dev: torch.randn(w, n + n % 2, dtype=dt, device=dev)[:, :n].t(),
    "odd columns": lambda n, w, dt, dev: torch.randn(w, n + 1 + n % 2, dtype=dt, device=dev)[:, 1:n + 1].t(),
    "every other": lambda n, w, dt, dev: torch.randn(n, 2 * w + 1, dtype=dt, device=dev)[:, :2 * w:2],
}
ROW_MAJOR = ("rows", "even pitch", "odd pitch", "unaligned")
WIDTHS = [(1, 9), (7, 5), (8, 8), (9, 1), (16, 17), (24, 24), (13, 37), (40, 20), (33, 7), (49, 57), (56, 56), (63, 64),
          (64, 3)]
ROWS = [1, 3, 63, 64, 65, 259, 4099]


def check(A, B, C, what):
    R = A.double().t() @ B.double()
    n = max(1, A.shape[0])
    bound = 4 * math.sqrt(n) * 2.0 ** -53 * float(A.double().norm()) * float(B.double().norm())
    err = (C.double() - R).abs()
    if C.dtype == torch.float32:
        err = (err - 2.0 ** -24 * R.abs() * (1 + 1e-6)).clamp_min(0)
    assert float(err.norm()) <= 2 * bound, (what, float(err.norm()), bound)  # 2: the reference has the same bound


def tile_index(dtype, m, k):
    from tsm_benchmark_b200 import variants
    hi, lo = (max(m, k) + 7) // 8 * 8, (min(m, k) + 7) // 8 * 8
    (i,) = [v["index"] for v in variants() if v["kind"] == "direct_dmma" and v["dtype"] == dtype
            and (v["wa"], v["wb"]) == (hi, lo)]
    return i


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("la,lb", list(itertools.product(ROW_MAJOR, ROW_MAJOR)))
def test_row_major(gpu, dtype, la, lb):
    from tsm_benchmark_b200 import tsmttsm, workspace_status
    dt = torch.float64 if dtype == "f64" else torch.float32
    torch.manual_seed(3)
    for m, k in WIDTHS:
        for n in ROWS:
            A, B = LAYOUTS[la](n, m, dt, gpu), LAYOUTS[lb](n, k, dt, gpu)
            check(A, B, tsmttsm(A, B, variant=tile_index(dtype, m, k)), (la, lb, n, m, k))
            if dtype == "f64":  # whichever kernel the rule picks (FP32 kernels sum in FP32)
                check(A, B, tsmttsm(A, B), ("default", la, lb, n, m, k))
    assert workspace_status(gpu) == 0


@pytest.mark.parametrize("la,lb", [(a, b) for a, b in itertools.product(LAYOUTS, LAYOUTS)
                                   if not (a in ROW_MAJOR and b in ROW_MAJOR)])
def test_any_strides(gpu, la, lb):
    from tsm_benchmark_b200 import tsmttsm, workspace_status
    torch.manual_seed(4)
    for m, k in WIDTHS:
        for n in (1, 2, 63, 66, 1001):
            A, B = LAYOUTS[la](n, m, torch.float64, gpu), LAYOUTS[lb](n, k, torch.float64, gpu)
            C = torch.ones((m, k), dtype=torch.float64, device=gpu)
            check(A, B, tsmttsm(A, B, C), (la, lb, n, m, k))
            C.fill_(1.0)
            check(A, B, tsmttsm(A, B, C, accumulate=True) - 1.0, ("accumulate", la, lb, n, m, k))
    assert workspace_status(gpu) == 0


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("gap", [-3, 0, 1, 2, 3, 7])
@pytest.mark.parametrize("pad", [0, 1, 4])
def test_neighbouring_column_blocks(gpu, dtype, gap, pad):
    """B's columns after A's (and A's after B's) in one matrix, overlapping
    (gap < 0), adjacent and apart; B = A."""
    from tsm_benchmark_b200 import tsmttsm
    dt = torch.float64 if dtype == "f64" else torch.float32
    torch.manual_seed(5)
    for m, k in WIDTHS:
        if m + gap < 0:
            continue
        for n in (5, 63, 200, 4099):
            V = torch.randn(n, pad + m + max(gap, 0) + k + pad, dtype=dt, device=gpu)
            X, Y = V[:, pad:pad + m], V[:, pad + m + gap:pad + m + gap + k]
            idx = tile_index(dtype, m, k)
            check(X, Y, tsmttsm(X, Y, variant=idx), ("after", gap, pad, n, m, k))
            check(Y, X, tsmttsm(Y, X, variant=idx), ("before", gap, pad, n, m, k))
            C = tsmttsm(X, X, variant=tile_index(dtype, m, m))
            check(X, X, C, ("itself", pad, n, m))
            assert torch.equal(C, C.t())


def test_repeatable(gpu):
    from tsm_benchmark_b200 import tsmttsm
    torch.manual_seed(6)
    V = torch.randn(300007, 50, dtype=torch.float64, device=gpu)
    A, B = V[:, 1:38], V[:, 38:]
    first = tsmttsm(A, B).clone()
    for _ in range(4):
        assert torch.equal(tsmttsm(A, B), first)


@pytest.mark.parametrize("n,m,k", [(1 << 18, 13, 13), (70001, 24, 20), (3001, 50, 50), (9000, 63, 60)])
def test_noalloc_takes_what_it_took(gpu, n, m, k):
    """The 4 MiB array holds a call if it holds one partial per CTA of the SIMT
    kernel's grid; the tile kernel then runs on a grid that fits."""
    from tsm_benchmark_b200 import _capi, variants
    lib = _capi.load()
    sh = int(torch.cuda.current_stream(gpu).cuda_stream)
    A = torch.randn(n, m, dtype=torch.float64, device=gpu)
    B = torch.randn(n, k, dtype=torch.float64, device=gpu)
    C = torch.empty(m, k, dtype=torch.float64, device=gpu)
    simt = [v for v in variants() if v["kind"] == "bulk" and v["dtype"] == "f64" and not v["exact"]
            and v["wa"] >= m and v["wb"] >= k][0]
    rows = n - n % (1 if (m % 2 == 0 and k % 2 == 0) else 2)
    sms = torch.cuda.get_device_properties(gpu).multi_processor_count
    ctas = max(1, min(-(-rows // simt["rows"]), sms))
    fits = 256 + ctas * m * k * 8 <= 4 << 20
    st = lib.tsm_gemm_tn_f64_noalloc(sh, n, m, k, A.data_ptr(), m, B.data_ptr(), k, C.data_ptr(), k, 0)
    assert (st == 0) == fits, (st, ctas)
    if fits:
        check(A, B, C, (n, m, k))
    else:
        assert st == 2  # TSM_ERROR_WORKSPACE


def test_infinities_stay_in_their_columns(gpu):
    """A padded column reads its neighbours' values: infinities and NaN must
    only reach the entries of C that hold them."""
    from tsm_benchmark_b200 import tsmttsm
    torch.manual_seed(7)
    V = torch.randn(5003, 21, dtype=torch.float64, device=gpu)
    V[17, 0] = float("inf")
    V[4000, 12] = float("nan")
    V[5002, 20] = float("-inf")
    A, B = V[:, 1:12], V[:, 13:20]
    check(A, B, tsmttsm(A, B), "neighbours outside")
    X = torch.randn(4097, 13, dtype=torch.float64, device=gpu)
    X[4096, 12] = float("inf")
    Y = torch.randn(4097, 11, dtype=torch.float64, device=gpu)
    C = tsmttsm(X, Y)
    assert bool(torch.isfinite(C[:12]).all()) and not bool(torch.isfinite(C[12]).any())
    assert np.isfinite(tsmttsm(Y, X)[:, :12].cpu().numpy()).all()
