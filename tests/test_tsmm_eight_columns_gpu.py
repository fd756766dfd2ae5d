"""FP32 Y = X W with 8 columns out of fewer, on either side of the size from
which the kernel for powers of two takes it, and the backward and accumulating
calls of the same widths, against FP64 with the bounds of test_tsmm_tile_gpu.py."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,q", [(7, 8), (5, 8), (1, 8), (8, 7)])
@pytest.mark.parametrize("side", [-1, 1])
def test_either_side(gpu, p, q, side):
    from tests.test_tsmm_tile_gpu import check
    from tsm_benchmark_b200 import tsmm, tsmttsm_backward, workspace_status
    torch.manual_seed(p + 64 * q)
    n = (8 << 20) // (4 * (p + q)) + 3 * side
    X = torch.randn(n, p, device=gpu)
    W = torch.randn(p, q, device=gpu)
    B = torch.randn(n, q, device=gpu)
    check(tsmm(X, W), X, W, None, "Y = X W")
    dX, dB = tsmttsm_backward(X, B, W)
    check(dX, B, W.t(), None, "dX")
    check(dB, X, W, None, "dB")
    Y = B.clone()
    tsmm(X, W, Y, accumulate=True)
    scale = float((X.abs() @ W.abs()).max() + B.abs().max())
    assert float((Y.double() - B.double() - X.double() @ W.double()).abs().max()) <= 2.0**-22 * scale
    assert workspace_status(gpu) == 0
