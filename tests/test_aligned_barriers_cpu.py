"""Barriers of the ``.aligned`` kind in the device sources: a warp has to come to them as one."""
import glob
import os
import re

from alpaca_lora_4bit_b200 import _lib

CSRC = os.path.join(os.path.dirname(_lib.__file__), "csrc")


def test_a_warp_meets_before_an_aligned_barrier():
    """The exchange of the weights-in-TMEM kernel was reached by warp 0 straight from a loop that its lane 0 runs alone: nothing
    but the compiler's choice of a meeting point brought the other lanes to the cluster's barrier together with it."""
    raw = re.compile(r'asm volatile\("(?:barrier\.cluster\.arrive[a-z.]*\.aligned|bar\.sync)')
    found = {}
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        text = open(path).read()
        found[os.path.basename(path)] = [text[:at.start()].rstrip().splitlines()[-1].strip() for at in raw.finditer(text)]
    assert found.pop("q4_async.cuh") == ["__syncwarp();"] * 2           # cluster_sync_all, named_bar_sync
    found.pop("q4_gemv.cu")                                              # (one of its own, in set-up code that no lane leaves)
    assert not any(found.values())
