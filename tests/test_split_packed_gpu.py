"""The TF32 split of narrow operands (several row groups share a tile) at the
edges of chunks, chunk pairs, slots and CTAs, against A^T B in FP64: 1e-6 of
sum |a| |b| per entry, the form's stated error."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k", [(1, 1), (1, 2), (3, 2), (5, 6), (7, 9), (10, 10), (11, 1), (15, 16), (3, 16), (17, 1)])
def test_narrow_widths(gpu, m, k):
    from tsm_benchmark_b200 import tsmttsm_split, workspace_status
    sms = torch.cuda.get_device_properties(gpu).multi_processor_count
    pack = 32 // max(m, k)
    whole = 64 * sms  # one chunk for every CTA
    ns = [1, 3, 5, 63, 64, 65, 129, whole - 1, whole, whole + 1, 2 * whole + 64, 3 * whole,
          2 * pack * whole - 64, 2 * pack * whole, 2 * pack * whole + 67, (2 * pack + 1) * whole + 1]
    torch.manual_seed(m + 40 * k)
    for n in ns:
        A = torch.randn(n, m, device=gpu)
        B = torch.randn(n, k, device=gpu)
        C = tsmttsm_split(A, B)
        Ad, Bd = A.double(), B.double()
        err = (C - Ad.t() @ Bd).abs() / (Ad.abs().t() @ Bd.abs())
        assert float(err.max()) <= 1e-6, (n, float(err.max()))
        assert torch.equal(C, tsmttsm_split(A, B)), n
    assert workspace_status(gpu) == 0


def test_infinities_stay_in_their_columns(gpu):
    from tsm_benchmark_b200 import tsmttsm_split
    torch.manual_seed(3)
    A, B = torch.randn(200001, 5, device=gpu), torch.randn(200001, 3, device=gpu)
    A[77777, 2] = float("inf")
    C = tsmttsm_split(A, B)
    keep = [0, 1, 3, 4]
    assert bool(torch.isfinite(C[keep]).all()) and not bool(torch.isfinite(C[2]).any())
