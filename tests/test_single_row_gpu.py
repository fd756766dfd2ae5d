"""One row, or none, has no row stride: any is taken, also one that no tensor map
could hold (2^40 bytes)."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1])
@pytest.mark.parametrize("m,k", [(1, 1), (5, 7), (8, 8), (13, 13), (24, 20), (37, 64), (3, 64)])
@pytest.mark.parametrize("ld", [64, 1 << 38, (1 << 38) + 1])
def test_any_row_stride(gpu, n, m, k, ld):
    from tsm_benchmark_b200 import _capi
    lib = _capi.load()
    A = torch.randn(1, m, dtype=torch.float64, device=gpu)
    B = torch.randn(1, k, dtype=torch.float64, device=gpu)
    ws = torch.zeros(lib.tsm_gemm_tn_workspace_size(n, m, k), dtype=torch.uint8, device=gpu)
    stream = torch.cuda.current_stream().cuda_stream
    want = A.t() @ B if n else torch.zeros(m, k, dtype=torch.float64, device=gpu)
    for call in ("plain", "strided"):
        C = torch.full((m, k), 7.0, dtype=torch.float64, device=gpu)
        args = (C.data_ptr(), k, 0, ws.data_ptr(), ctypes.c_size_t(ws.numel()))
        if call == "plain":
            st = lib.tsm_gemm_tn_f64(stream, n, m, k, A.data_ptr(), ld, B.data_ptr(), ld, *args)
        else:
            st = lib.tsm_gemm_tn_strided_f64(stream, n, m, k, A.data_ptr(), ld, 1, B.data_ptr(), ld, 1, *args)
        assert st == 0, (call, lib.tsm_last_cuda_error())
        assert torch.allclose(C, want, rtol=1e-15, atol=0), call
