"""The cross-CTA sum at the edges of its two levels: one group up to 32 CTAs
(64 where m*k <= 256), groups of ceil(sqrt(G)) beyond, odd and even m*k, a ragged last group."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctas", [1, 2, 16, 17, 31, 32, 33, 37, 64, 65, 144, 145, 148])
@pytest.mark.parametrize("m,k", [(3, 5), (8, 8), (64, 64)])
def test_grid_sizes(gpu, oracle_mod, ctas, m, k):
    from tsm_benchmark_b200 import _capi
    n = 148 * 520
    A, B = oracle_mod.operands(n, m, k, seed=ctas + m)
    dA, dB = torch.from_numpy(A).to(gpu), torch.from_numpy(B).to(gpu)
    lib = _capi.load()
    need = lib.tsm_gemm_tn_workspace_size(n, m, k)
    ws = torch.zeros(need, dtype=torch.uint8, device=gpu)
    sh = int(torch.cuda.current_stream(gpu).cuda_stream)
    got = []
    for accumulate in (0, 1):  # the second call finds the counters the first one left
        C = torch.ones((m, k), dtype=torch.float64, device=gpu)
        st = lib.tsm_gemm_tn_f64_launch(sh, n, m, k, dA.data_ptr(), m, dB.data_ptr(), k, C.data_ptr(), k, accumulate,
                                        ws.data_ptr(), need, -1, ctas)
        assert st == 0
        got.append(C.cpu().numpy() - accumulate)
    ref = oracle_mod.naive(A, B)
    for C in got:
        nw = oracle_mod.normwise(A, B, ref, C)
        assert nw["err"] <= nw["bound"], (ctas, m, k, nw)
    assert int(ws[:256].to(torch.int32).sum()) == 0  # counters and error word back to zero
