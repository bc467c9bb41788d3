"""Loads from another block's shared memory are ordered by the cluster barrier in front of them only where the compiler may not move them: an ``asm`` that reads
``shared::cluster`` without being volatile, or without clobbering memory, may be lifted over the barrier.  Read from the sources, so that it needs no GPU."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mini_inference_engine_b200", "csrc")


def loads():
    """(file, line, statement) of every ``asm`` of the package that loads from a cluster's shared memory."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = open(path).read()
        for m in re.finditer(r"\basm\b[^;]*?\"\s*ld\.shared::cluster(?:\\.|[^\"\\])*\"[^;]*;", text):
            yield os.path.basename(path), text[:m.start()].count("\n") + 1, m.group(0)


def test_cluster_loads_stay_behind_the_barrier():
    found = list(loads())
    assert found                                       # (the pattern still meets the helpers)
    moved = [f"{name}:{line}" for name, line, text in found if not re.match(r"asm\s+volatile\b", text) or not re.search(r":\s*\"memory\"\s*\)\s*;$", text)]
    assert not moved, moved
