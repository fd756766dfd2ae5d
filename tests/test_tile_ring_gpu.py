"""The tile kernels' ring beyond its first round: stages used again, barrier
phases, the slots' turns and the units' turns across chunks, several boxes a
chunk.  With a grid of one or two CTAs a few thousand rows are many chunks; where
the call has no grid to cap, the rows are many.  Against FP64, with the bounds of
test_tile_gpu.py and test_tsmm_tile_gpu.py."""
import pytest
import torch

from tests.test_tile_gpu import LAYOUTS, ROW_MAJOR, check, tile_index

pytestmark = pytest.mark.gpu

PAIRS = [(1, 9), (7, 5), (13, 13), (24, 8), (40, 20), (64, 57)]


def launch(A, B, max_ctas):
    """C = A^T B on the tile kernel with at most max_ctas CTAs."""
    from tsm_benchmark_b200 import _capi
    from tsm_benchmark_b200.api import workspace
    lib = _capi.load()
    (n, m), k = A.shape, B.shape[1]
    C = torch.empty((m, k), dtype=torch.float64, device=A.device)
    stream = torch.cuda.current_stream().cuda_stream
    ws = workspace(A.device, lib.tsm_gemm_tn_workspace_size(n, m, k), torch.cuda.current_stream())
    st = lib.tsm_gemm_tn_f64_launch(stream, n, m, k, A.data_ptr(), A.stride(0), B.data_ptr(), B.stride(0),
                                    C.data_ptr(), k, 0, ws.data_ptr(), ws.numel(), tile_index("f64", m, k), max_ctas)
    assert st == 0
    return C


@pytest.mark.parametrize("layout", [*ROW_MAJOR, "joint", "joint, odd pitch", "joint, unaligned"])
@pytest.mark.parametrize("m,k", PAIRS)
def test_many_chunks_a_cta(gpu, layout, m, k):
    from tsm_benchmark_b200 import workspace_status
    torch.manual_seed(m + 64 * k)
    for n, ctas in ((4 * 1024 + 5, 1), (20011, 1), (30001, 2)):
        if layout.startswith("joint"):
            ld = {"joint": m + k + (m + k) % 2, "joint, odd pitch": (m + k) | 1, "joint, unaligned": m + k + 2}[layout]
            first = 1 if layout == "joint, unaligned" else 0
            V = torch.randn(n * ld + 1, dtype=torch.float64, device=gpu)[first:first + n * ld].view(n, ld)
            A, B = V[:, :m], V[:, m:m + k]
        else:
            A, B = LAYOUTS[layout](n, m, torch.float64, gpu), LAYOUTS[layout](n, k, torch.float64, gpu)
        check(A, B, launch(A, B, ctas), (layout, m, k, n, ctas))
    assert workspace_status(gpu) == 0


@pytest.mark.parametrize("dtype,layout", [*((d, x) for d in (torch.float64, torch.float32) for x in ROW_MAJOR),
                                          *((torch.float64, x) for x in ("columns", "odd columns", "mixed"))])
@pytest.mark.parametrize("m,k", [(1, 2), (5, 8), (13, 8), (24, 9)])
def test_many_chunks_on_the_whole_grid(gpu, dtype, layout, m, k):
    from tsm_benchmark_b200 import tsmttsm, workspace_status
    torch.manual_seed(m + 64 * k)
    n = 4 * 148 * 1024 + 77  # four chunks of the longest kind a CTA
    A = LAYOUTS["odd columns" if layout == "mixed" else layout](n, m, dtype, gpu)
    B = LAYOUTS["rows" if layout == "mixed" else layout](n, k, dtype, gpu)
    variant = tile_index("f64" if dtype == torch.float64 else "f32", m, k) if layout in ROW_MAJOR else -1
    check(A, B, tsmttsm(A, B, variant=variant), (layout, m, k))
    assert workspace_status(gpu) == 0


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("p,q", [(1, 1), (3, 3), (2, 4), (7, 5), (6, 7), (5, 9), (13, 3)])
def test_tsmm_many_chunks(gpu, dtype, p, q):
    from tests.test_tsmm_tile_gpu import check as check_rows
    from tsm_benchmark_b200 import tsmm, workspace_status
    torch.manual_seed(p + 64 * q)
    n = 6 * 148 * 2048 + 45  # six chunks of the longest kind a CTA, four stages
    X = torch.randn(n, p, dtype=dtype, device=gpu)
    W = torch.randn(p, q, dtype=dtype, device=gpu)
    check_rows(tsmm(X, W), X, W, None, (p, q))
    Y = torch.randn(n, q, dtype=dtype, device=gpu)
    old = Y.clone()
    tsmm(X, W, Y, accumulate=True)
    if dtype == torch.float64:
        check_rows(Y, X, W, old, (p, q, "+="))
    else:  # an unaligned remainder of rows adds in FP32: two roundings
        scale = float((X.abs() @ W.abs()).max() + old.abs().max())
        assert float((Y.double() - old.double() - X.double() @ W.double()).abs().max()) <= 2.0**-22 * scale
    assert workspace_status(gpu) == 0


def test_repeated_bits_are_the_product(gpu):
    """The call test_tile_gpu.py repeats for equal bits, against FP64."""
    from tsm_benchmark_b200 import tsmttsm
    torch.manual_seed(6)
    V = torch.randn(300007, 50, dtype=torch.float64, device=gpu)
    A, B = V[:, 1:38], V[:, 38:]
    check(A, B, tsmttsm(A, B), "repeat")
