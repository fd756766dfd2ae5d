"""Large operands of at most 8 columns whose strides no tensor map describes: on
either side of the sizes and widths where the direct-load kernel takes them,
against A^T B in FP64 (4 sqrt(n) 2^-53 ||A|| ||B|| for each side)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

LINE = 30 << 20  # bytes from which the direct kernel is considered


def columns(n, w, dev):  # odd column pitch
    ld = n | 1
    return torch.randn(w * ld, dtype=torch.float64, device=dev).as_strided((n, w), (1, ld))


def two_strides(n, w, dev):
    return torch.randn(n, 2 * w + 1, dtype=torch.float64, device=dev)[:, :2 * w:2]


def rows(n, w, dev):
    return torch.randn(n, w, dtype=torch.float64, device=dev)


@pytest.mark.parametrize("kinds", [(columns, columns), (two_strides, two_strides), (columns, two_strides),
                                   (rows, columns), (columns, rows)])
@pytest.mark.parametrize("m,k", [(8, 8), (7, 7), (6, 7), (5, 5), (5, 3), (4, 6), (8, 1), (1, 8)])
def test_on_either_side_of_the_line(gpu, kinds, m, k):
    from tsm_benchmark_b200 import tsmttsm, workspace_status
    torch.manual_seed(m + 64 * k)
    for n in (LINE // (8 * (m + k)) - 1, (LINE // (8 * (m + k)) + 2) | 1):
        A, B = kinds[0](n, m, gpu), kinds[1](n, k, gpu)
        C0 = torch.randn(m, k, dtype=torch.float64, device=gpu)
        got = tsmttsm(A, B, C0.clone(), accumulate=True) - C0
        bound = 4 * math.sqrt(n) * 2.0**-53 * float(A.norm()) * float(B.norm())
        assert float((got - A.t() @ B).norm()) <= 2 * bound, (kinds, n)
        assert torch.equal(tsmttsm(A, B), tsmttsm(A, B))
    assert workspace_status(gpu) == 0


def test_a_matrix_with_itself_is_symmetric(gpu):
    from tsm_benchmark_b200 import tsmttsm
    A = columns(300001, 8, gpu)
    C = tsmttsm(A, A)
    assert torch.equal(C, C.t())
