"""Every place where one lane acquires a progress counter and hands it to its warp by a shuffle has
a __syncwarp() before the warp goes on: a shuffle orders no memory, so without it the other lanes'
reads of the rows behind the counter are not ordered after the acquire.  Read from the sources (a
machine that happens to order the reads would not show it)."""

import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pyalign_gb300", "csrc")


def broadcasts(text):
    """(line, code up to the next return or read of a row) of each shuffle of an acquired value."""
    for m in re.finditer(r"\b(\w+) = (?:ld_acquire|wait_progress)\(", text):
        tail = text[m.end():m.end() + 600]
        s = re.search(r"= __shfl_sync\(0xffffffffu, " + m.group(1) + r", 0\);", tail)
        if not s or "__ldcg" in tail[:s.start()]:
            continue
        rest = tail[s.end():]
        stop = re.search(r"\breturn\b|__ldcg|\n\t*}\n", rest)
        yield text.count("\n", 0, m.end() + s.end()) + 1, rest[:stop.start() if stop else len(rest)]


def test_acquired_counters_are_ordered_before_the_warps_reads():
    found = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for line, code in broadcasts(text):
            found += 1
            assert "__syncwarp()" in code, (os.path.basename(path), line)
    assert found >= 3  # the chunked rows of the chained kernels, the finished tiles of general gaps
