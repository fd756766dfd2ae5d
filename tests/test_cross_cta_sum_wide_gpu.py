"""The cross-CTA sum of wide products on few CTAs, where a thread sums four
entries at once: grids from one CTA to past the second level, against FP64
(4 sqrt(n) 2^-53 ||A|| ||B|| for each side), with a Gram matrix exactly symmetric."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def launch(A, B, C, accumulate, max_ctas):
    from tsm_benchmark_b200 import _capi
    from tsm_benchmark_b200.api import workspace
    lib = _capi.load()
    (n, m), k = A.shape, B.shape[1]
    ws = workspace(A.device, lib.tsm_gemm_tn_workspace_size(n, m, k), torch.cuda.current_stream())
    st = lib.tsm_gemm_tn_f64_launch(torch.cuda.current_stream().cuda_stream, n, m, k, A.data_ptr(), m, B.data_ptr(), k,
                                    C.data_ptr(), k, accumulate, ws.data_ptr(), ws.numel(), -1, max_ctas)
    assert st == 0
    return C


@pytest.mark.parametrize("m,k", [(64, 64), (57, 63), (48, 64), (33, 40), (32, 32), (64, 16)])
@pytest.mark.parametrize("ctas", [1, 2, 3, 4, 5, 8, 12, 13, 16, 17, 21, 32, 33, 50, 148])
def test_any_grid(gpu, m, k, ctas):
    torch.manual_seed(m + 64 * k + ctas)
    n = 200 * ctas + 3
    A = torch.randn(n, m, dtype=torch.float64, device=gpu)
    B = torch.randn(n, k, dtype=torch.float64, device=gpu)
    C0 = torch.randn(m, k, dtype=torch.float64, device=gpu)
    bound = 4 * math.sqrt(n) * 2.0**-53 * float(A.norm()) * float(B.norm())
    for acc in (0, 1):
        got = launch(A, B, C0.clone(), acc, ctas)
        assert float((got - A.t() @ B - (C0 if acc else 0)).norm()) <= 2 * bound, acc
    if m == k:
        got = launch(A, A, C0.clone(), 0, ctas)
        assert torch.equal(got, got.t())
        assert float((got - A.t() @ A).norm()) <= 2 * 4 * math.sqrt(n) * 2.0**-53 * float(A.norm()) ** 2
