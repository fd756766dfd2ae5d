"""Y = X W, Y += X W and the fused backward for widths that are not powers of
two, at the edges of 4-column k-steps, 8-column tiles, 16- and 32-row units and
chunks, against the same products in FP64.

Each entry is a sum of p products: |error| <= (p + 2) 2^-53 (|X| |W| + |Y0|) in
FP64, plus one rounding to FP32 (2^-24 of the entry) where the storage is FP32;
twice that, since the reference has the same error."""
import pytest
import torch

pytestmark = pytest.mark.gpu

WIDTHS = [(1, 1), (1, 7), (3, 3), (4, 5), (5, 8), (8, 9), (7, 16), (13, 13), (17, 4), (20, 40), (24, 24), (37, 13),
          (33, 33), (48, 48), (5, 60), (63, 63), (64, 1), (64, 57)]
ROWS = [1, 2, 3, 4, 15, 31, 32, 33, 65, 1000, 4099, 40007]


def check(got, X, W, Y0, what):
    X, W = X.double(), W.double()
    ref, size = X @ W, X.abs() @ W.abs()
    if Y0 is not None:
        ref, size = ref + Y0.double(), size + Y0.double().abs()
    tol = 2 * (X.shape[1] + 2) * 2.0 ** -53 * size
    if got.dtype == torch.float32:
        tol = tol + 2.0 ** -24 * (1 + 1e-6) * ref.abs()
    bad = (got.double() - ref).abs() > tol
    assert not bool(bad.any()), (what, int(bad.sum()))


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("m,k", WIDTHS)
def test_backward_and_accumulate(gpu, dtype, m, k):
    from tsm_benchmark_b200 import tsmm, tsmttsm_backward, workspace_status
    torch.manual_seed(m + 100 * k)
    for n in ROWS:
        A = torch.randn(n, m, dtype=dtype, device=gpu)
        B = torch.randn(n, k, dtype=dtype, device=gpu)
        W = torch.randn(m, k, dtype=dtype, device=gpu)
        dA, dB = tsmttsm_backward(A, B, W)
        check(dA, B, W.t(), None, ("dA", n))
        check(dB, A, W, None, ("dB", n))
        # guard rows: the store of whole chunks must end with the last row
        buf = torch.randn(n + 2, k, dtype=dtype, device=gpu)
        old = buf.clone()
        Y = buf[:n]
        tsmm(A, W, Y, accumulate=True)
        if dtype == torch.float64:
            check(Y, A, W, old[:n], ("Y", n))
        else:  # an unaligned remainder of rows adds in FP32: two roundings
            assert torch.allclose(Y.double(), old[:n].double() + A.double() @ W.double(), rtol=2.0 ** -22,
                                  atol=2.0 ** -22 * float((A.abs() @ W.abs()).max() + old.abs().max()))
        assert torch.equal(buf[n:], old[n:]), ("guard", n)
    assert workspace_status(gpu) == 0


@pytest.mark.parametrize("m,k", [(13, 13), (24, 20), (63, 5)])
def test_special_values_stay_in_their_rows(gpu, m, k):
    """Columns past p read the next row's values: an infinity there must not
    reach this row."""
    from tsm_benchmark_b200 import tsmm
    torch.manual_seed(1)
    X = torch.randn(517, m, dtype=torch.float64, device=gpu)
    W = torch.randn(m, k, dtype=torch.float64, device=gpu)
    ref = X @ W
    X[100] = float("inf")
    X[101, 0] = float("nan")
    Y = tsmm(X, W)
    keep = torch.ones(517, dtype=torch.bool, device=gpu)
    keep[100:102] = False
    assert bool(torch.isfinite(Y[keep]).all()) and torch.allclose(Y[keep], ref[keep], rtol=1e-12, atol=1e-12)
    assert bool(torch.isnan(Y[101]).all()) and not bool(torch.isfinite(Y[100]).any())


def test_repeatable_on_two_streams(gpu):
    from tsm_benchmark_b200 import tsmttsm_backward
    torch.manual_seed(2)
    A = torch.randn(200003, 24, dtype=torch.float64, device=gpu)
    B = torch.randn(200003, 10, dtype=torch.float64, device=gpu)
    W = torch.randn(24, 10, dtype=torch.float64, device=gpu)
    first = tsmttsm_backward(A, B, W)
    torch.cuda.synchronize()
    side = [torch.cuda.Stream(gpu) for _ in range(2)]
    got = [tsmttsm_backward(A, B, W, stream=s) for s in side for _ in range(3)]
    torch.cuda.synchronize()
    for dA, dB in got:
        assert torch.equal(dA, first[0]) and torch.equal(dB, first[1])
