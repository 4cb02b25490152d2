"""The build compares its objects with every file a translation unit includes."""

import os
import re

from pyalign_gb300 import build


def test_every_included_file_counts(monkeypatch):
    included = set()
    for f in os.listdir(build.CSRC):
        with open(os.path.join(build.CSRC, f)) as text:
            included |= {os.path.basename(x) for x in re.findall(r'#include "([^"]+)"', text.read())}
    times = {}
    monkeypatch.setattr(os.path, "getmtime", lambda p: times.setdefault(os.path.basename(p), 1.0))
    for f in sorted(included):
        times.clear()
        times[f] = 2.0
        assert build._deps() == 2.0, f
