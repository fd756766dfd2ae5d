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


def _enclosing(code, at):
    """Headers of the blocks around position `at`, innermost first."""
    depth = 0
    for i in range(at - 1, -1, -1):
        if code[i] == "}":
            depth += 1
        elif code[i] == "{":
            if depth:
                depth -= 1
                continue
            start = max(code.rfind(c, 0, i) for c in "{}") + 1
            yield code[start:i]


def test_a_warp_gives_up_a_wait_as_one():
    """A bounded wait of one lane (dev::mbar_wait) stands only where one lane
    runs, or where a lane that gave up stays in the loop, or stands in at its
    __syncwarps; else warps wait with one verdict (dev::mbar_wait_warp), or that lane would leave
    the others at the next warp-wide instruction."""
    single = re.compile(r"lane == 0|\bbool cm_produce\(|\bvoid cm_drain\(")
    seen = 0
    for f in glob.glob(os.path.join(CSRC, "*.cuh")):
        code = _code(f)
        for m in re.finditer(r"dev::mbar_wait\(", code):
            seen += 1
            statement = code[max(code.rfind(c, 0, m.start()) for c in ";{}") + 1:m.start()]
            heads = [statement, *_enclosing(code, m.start())]
            stands_in = re.search(r"^[^{}]*\{[^}]*for \(; (?:it|c) < [^)]*\) __syncwarp\(\);\s*break;",
                                  code[m.end():])
            stays = re.search(r"if \(ok && !$", code[:m.start()]) and re.match(
                r"[^{}]*\{\s*ok = false;\s*\*abort = 1;\s*atomicOr\([^;]*;\s*\}", code[m.end():])
            assert stands_in or stays or any(single.search(h.split(";")[-1]) for h in heads), (
                os.path.basename(f), code[m.start() - 80:m.end() + 60])
    assert seen >= 20
