"""Y = X W on the rows and widths the power-of-two TSMM kernels guard: the
last, partial chunk at p = 4, and every chunk of other widths with a pitched Y
(a column block of a wider matrix), against FP64."""
import pytest
import torch

from tsm_benchmark_b200 import tsmm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("n,p,q,pitched", [
    (5, 4, 4, False), (37, 4, 16, False), (1000, 4, 8, False), (40007, 4, 4, False), (200003, 4, 32, False),
    (37, 3, 5, True), (1000, 4, 4, True), (4099, 6, 7, True), (4099, 13, 13, True), (40007, 24, 9, True),
    (40007, 1, 3, True), (4099, 37, 13, True), (4099, 63, 64, True),
])
def test_guarded_rows(gpu, n, p, q, pitched, accumulate, dtype):
    g = torch.Generator(device="cuda").manual_seed(n + 64 * p + q)

    def rand(*shape):
        return torch.empty(shape, dtype=dtype, device=gpu).uniform_(-1, 1, generator=g)

    X, W = rand(n, p), rand(p, q)
    wide = rand(n, q + 3)
    Y = wide[:, :q] if pitched else wide[:, :q].contiguous()
    old = Y.clone().double()
    side = wide[:, q:].clone()
    tsmm(X, W, Y, accumulate=accumulate)
    want = X.double() @ W.double() + (old if accumulate else 0)
    # p products and sums in FP64 on either side, then one rounding to the
    # storage type (two where the old value is added in it)
    mag = X.double().abs() @ W.double().abs() + old.abs()
    eps = torch.finfo(dtype).eps
    bound = 2 * (p + 2) * 2.0**-53 * mag + (eps * mag if dtype == torch.float32 else 0)
    assert bool(((Y.double() - want).abs() <= bound).all())
    assert torch.equal(wide[:, q:], side)
