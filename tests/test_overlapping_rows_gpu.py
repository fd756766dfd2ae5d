"""Operands whose rows overlap: FP64 products take windows over a series
(``unfold``) as they lie, everything else asks for a copy."""
import pytest
import torch

import tsm_benchmark_b200 as tsm
from tsm_benchmark_b200.autograd import gram_tn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,step", [(2, 8, 1), (100, 8, 1), (5000, 8, 3), (5000, 13, 1), (20011, 16, 15)])
def test_windows_equal_their_copy(gpu, n, m, step):
    g = torch.Generator(device="cuda").manual_seed(n + m)
    x = torch.empty((n - 1) * step + m, dtype=torch.float64, device=gpu).uniform_(-1, 1, generator=g)
    W = x.unfold(0, m, step)
    B = torch.empty((n, 5), dtype=torch.float64, device=gpu).uniform_(-1, 1, generator=g)
    assert W.shape == (n, m)
    Wc = W.contiguous()
    for got, P, Q in ((tsm.tsmttsm(W, B), Wc, B), (tsm.tsmttsm(B, W), B, Wc), (tsm.tsmttsm(W, W), Wc, Wc)):
        # sums of n products in FP64 on either side
        bound = 2 * n * 2.0**-53 * (P.abs().t() @ Q.abs())
        assert bool(((got - P.t() @ Q).abs() <= bound).all())


def test_rows_that_overlap_are_refused(gpu):
    x = torch.zeros(64, dtype=torch.float64, device=gpu)
    B = torch.zeros((20, 8), dtype=torch.float64, device=gpu)
    same, windows = x[:8].expand(20, 8), x.unfold(0, 8, 1)[:20]
    C = torch.zeros((8, 8), dtype=torch.float64, device=gpu)
    with pytest.raises(ValueError):
        tsm.tsmttsm(same, B)
    for v in (same, windows):
        for call in (lambda: tsm.gram(v), lambda: tsm.block_orthogonalize(v, B), lambda: tsm.block_orthogonalize(B, v),
                     lambda: tsm.tsmm(v, C), lambda: tsm.tsmm(B, C, v), lambda: tsm.tsmttsm_backward(v, B, C),
                     lambda: tsm.tsmttsm_backward(B, v, C), lambda: tsm.tsmttsm(v.float()[:1].expand(20, 8), B.float()),
                     lambda: tsm.tsmttsm_split(x.float().unfold(0, 8, 1)[:20], B.float()),
                     lambda: tsm.tsmttsm(B, B, x[:8].expand(8, 8))):
            with pytest.raises(ValueError, match="overlap"):
                call()


def test_gradients_through_them(gpu):
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.empty(4106, dtype=torch.float64, device=gpu).uniform_(-1, 1, generator=g).requires_grad_()
    b = torch.empty((1, 4), dtype=torch.float64, device=gpu).uniform_(-1, 1, generator=g).requires_grad_()

    def loss(product):
        return product(x.unfold(0, 11, 1), b.expand(4096, 4)).square().sum()

    got = torch.autograd.grad(loss(gram_tn), (x, b))
    want = torch.autograd.grad(loss(lambda A, B: A.t() @ B), (x, b))
    for p, q in zip(got, want):
        assert torch.allclose(p, q, rtol=1e-10, atol=1e-10 * float(q.abs().max()))
