"""Which kernel a plain call takes, asked of the library without a GPU (the fake
addresses are never read): the tuning table, timed on dense aligned rows, does
not decide for column slices, odd pitches and unaligned rows."""
import functools
import itertools

import pytest

BASE = 1 << 20
ROWS = [1 << 12, 1 << 16, 1 << 20, 1 << 24]
PAIRS = [(m, k) for m, k in itertools.product((1, 2, 4, 8, 16, 32, 48, 64), repeat=2)]


def operands(layout, n, m, k):
    """(A, lda, B, ldb) as byte addresses and pitches of FP64 operands."""
    far = BASE + (1 << 40)
    return {"neighbours": (BASE, m + k + (m + k) % 2, BASE + 8 * m, m + k + (m + k) % 2),
            "neighbours, odd pitch": (BASE, m + k + 1 + (m + k) % 2, BASE + 8 * m, m + k + 1 + (m + k) % 2),
            "odd pitch": (BASE, m + 1 + m % 2, far + 8, k + 1 + k % 2),
            "unaligned": (BASE + 8, m, far + 8, k)}[layout]


@functools.cache
def table():
    from tsm_benchmark_b200 import variants
    return variants()


def default(n, m, k, A, lda, B, ldb):
    from tsm_benchmark_b200 import _capi
    return table()[_capi.load().tsm_gemm_tn_default_variant(0, n, m, k, A, lda, B, ldb)]


@pytest.mark.parametrize("layout", ["neighbours", "neighbours, odd pitch", "odd pitch", "unaligned"])
def test_both_orders_take_the_same_way(layout):
    """No table entry decides for these rows, so m x k and k x m agree, and a
    direct kernel is the one with the least capacities."""
    for (m, k), n in itertools.product(PAIRS, ROWS):
        v, w = (default(n, a, b, *operands(layout, n, a, b)) for a, b in ((m, k), (k, m)))
        if "dmma" in (v["kind"], w["kind"]):  # tensor boxes: any 16-byte pitch, tuned per pair
            assert min(m, k) >= 16 and layout == "neighbours", (m, k, n, v["name"])
            continue
        assert v["kind"] == w["kind"], (layout, m, k, n, v["name"], w["name"])
        if v["kind"] == "direct":
            least = tuple(64 if x == 48 else x for x in (m, k))
            assert (v["wa"], v["wb"]) == least, (layout, m, k, n, v["name"])


@pytest.mark.parametrize("n", [1 << 20, 1 << 24])
def test_wide_neighbours_on_the_tile_kernel_narrow_slices_apart_direct(n):
    for m, k in [(8, 32), (4, 32), (4, 16), (1, 64), (16, 8)]:
        for layout in ("neighbours", "neighbours, odd pitch"):
            assert default(n, m, k, *operands(layout, n, m, k))["kind"] == "direct_dmma", (layout, m, k)
    for m, k in [(8, 4), (4, 8), (16, 4), (4, 4)]:
        for layout in ("odd pitch", "unaligned"):
            assert default(n, m, k, *operands(layout, n, m, k))["kind"] == "direct", (layout, m, k)


def test_dense_rows_keep_the_table():
    import json
    import os

    from tests.conftest import ROOT
    with open(os.path.join(ROOT, "tsm_benchmark_b200", "tuned.json")) as f:
        choices = json.load(f)["choices"]
    for c in choices:
        m, k = c["m"], c["k"]
        later = [d["nmin"] for d in choices if (d["m"], d["k"]) == (m, k) and d["nmin"] > c["nmin"]]
        for n in [max(1, c["nmin"]), *[x - 1 for x in later[:1]]]:
            v = default(n, m, k, BASE, m, BASE + (1 << 40), k)
            assert v["name"] == c["variant"], (m, k, n, v["name"], c["variant"])
