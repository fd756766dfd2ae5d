"""A^T A of pitched rows: which kernel it takes (asked of the library without a GPU;
the address is never read)."""
import pytest


@pytest.mark.parametrize("m", range(1, 65))
def test_half_filled_boxes_of_large_operands_stay_direct(m):
    from tsm_benchmark_b200 import _capi, variants
    lib, table = _capi.load(), variants()
    A, pitch = 1 << 20, m + 2 + m % 2

    def kind(dtype, nbytes, size):
        return table[lib.tsm_gemm_tn_default_variant(dtype, nbytes // (size * m), m, m, A, pitch, A, pitch)]["kind"]

    if m % 16 == 0 and m > 8:
        assert kind(0, 300 << 20, 8) == "dmma"
        return
    assert kind(0, 300 << 20, 8) == ("direct" if m <= 6 else "direct_dmma")
    assert kind(0, 60 << 20, 8) == ("direct" if m < 5 else "direct_dmma")
    assert kind(1, 300 << 20, 4) == ("direct" if m < 5 else "direct_dmma")  # FP32: sums in FP64
