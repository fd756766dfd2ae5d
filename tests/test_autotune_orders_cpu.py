"""The autotuner's candidates do not depend on the order of the widths: the
any-layout tensor-core kernels take m x k and k x m (no GPU)."""
import json
import os

import pytest

from tests.conftest import ROOT

PAIRS = [(1, 64), (4, 16), (4, 32), (8, 16), (8, 32), (16, 32), (16, 64), (32, 48), (48, 64), (64, 64), (5, 37)]


@pytest.mark.parametrize("m,k", PAIRS)
def test_one_tile_candidate_in_either_order(m, k):
    from tsm_benchmark_b200 import variants
    from tsm_benchmark_b200.autotune import candidates
    vs = variants()
    tiles = [[v["name"] for v in candidates(vs, *pair) if v["kind"] == "direct_dmma"] for pair in ((m, k), (k, m))]
    hi, lo = (-(-w // 8) * 8 for w in (max(m, k), min(m, k)))
    assert tiles[0] == tiles[1] == [f"direct_dmma_{hi}x{lo}_cap"]


def test_tuned_pairs_with_the_narrower_operand_first_were_timed_against_the_tile_kernel():
    from tsm_benchmark_b200 import variants
    from tsm_benchmark_b200.autotune import candidates
    vs = variants()
    with open(os.path.join(ROOT, "tsm_benchmark_b200", "tuned.json")) as f:
        doc = json.load(f)
    for c in doc["choices"]:
        m, k = c["m"], c["k"]
        if -(-m // 8) >= -(-k // 8):
            continue
        (tile,) = [v["name"] for v in candidates(vs, m, k) if v["kind"] == "direct_dmma"]
        row = doc["timings"][f"{m}x{k}@{c['n_timed']}"]
        assert tile in row and row[tile]["ok"], (m, k, c["n_timed"])
