"""Barriers of the ``.aligned`` kind in the device sources: a warp has to come to them as one."""
import glob
import os
import re

from alpaca_lora_4bit_b200 import _lib

CSRC = os.path.join(os.path.dirname(_lib.__file__), "csrc")


def test_a_warp_meets_before_an_aligned_barrier():
    """The exchange of the weights-in-TMEM kernel was reached by warp 0 straight from a loop that its lane 0 runs alone: nothing
    but the compiler's choice of a meeting point brought the other lanes to the cluster's barrier together with it."""
    raw = re.compile(r"barrier\.cluster\.arrive|\bbar\.sync|\bnamed_bar_sync\(")
    found = {}
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        lines = open(path).read().splitlines()
        found[os.path.basename(path)] = {line.strip(): lines[i - 1].strip() for i, line in enumerate(lines) if raw.search(line)}
    helpers = found.pop("q4_async.cuh")
    assert [above for line, above in helpers.items() if "barrier.cluster" in line or line == "named_bar_sync(id, threads);"] == ["__syncwarp();"] * 2
    found.pop("q4_gemv.cu")                                  # decode: lanes part for single instructions only
    assert not any(found.values()), found
