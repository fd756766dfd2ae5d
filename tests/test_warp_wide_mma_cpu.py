"""The warp-wide instructions of the FP64 tensor-core kernels, checked in their
source (no GPU): a lane that branches around a load directly before an
``mma.sync`` can bring its warp to it in two parts, which never end, so the
kernels load from a valid address and select."""
import glob
import os
import re

from tests.conftest import ROOT

CSRC = os.path.join(ROOT, "tsm_benchmark_b200", "csrc")


def _code(path):
    return re.sub(r"//[^\n]*", "", open(path).read())


def test_no_conditional_load_in_the_mma_kernels():
    files = [f for f in glob.glob(os.path.join(CSRC, "*.cuh")) if "dmma_m8n8k4" in _code(f)]
    assert len(files) >= 5
    load = re.compile(r"\?\s*(?:static_cast<double>\()?\s*(?:x\w*|y\w*|s[ab]|stage)\s*(?:\[[^\]]*\])?\s*\[")
    for f in files:
        hits = [m.group(0) for m in load.finditer(_code(f))]
        assert not hits, (os.path.basename(f), hits)
