"""FP32 products of dense rows: which widths take the tensor-core tile kernel
(asked of the library without a GPU; the addresses are never read)."""
import functools

import pytest

BASE, N = 1 << 20, 1 << 20


@functools.cache
def table():
    from tsm_benchmark_b200 import variants
    return variants()


def kind(m, k):
    from tsm_benchmark_b200 import _capi
    v = table()[_capi.load().tsm_gemm_tn_default_variant(1, N, m, k, BASE, m, BASE + (1 << 40), k)]
    return "exact" if v["exact"] else v["kind"]


@pytest.mark.parametrize("hi", range(5, 65))
def test_eight_columns_a_thread_on_either_side(hi):
    """From 5 columns on a SIMT thread holds 8 of either side: no width in
    between stands out."""
    for lo in range(5, min(hi, 12) + 1):
        for m, k in ((lo, hi), (hi, lo)):
            assert kind(m, k) in ("direct_dmma", "exact"), (m, k)


def test_narrow_sides_by_banks_and_padding():
    for lo in (1, 2, 3, 4):
        for hi in range(16, 65):
            banks = hi % 8 == 0
            padding = lo >= 3 and 16 < hi <= 48
            for m, k in ((lo, hi), (hi, lo)):
                if kind(m, k) != "exact":
                    assert (kind(m, k) == "direct_dmma") == (banks or padding), (m, k)
