"""Path counts along the band of co-optimal paths, and the search for the first alignments
(need a GPU).

path_count_band_kernel counts forward from the one seed of a Global/Semiglobal pair; the
kernels over whole matrices (PA_COUNT_MODE=group, chain) count every cell.  The counts are
whole numbers and saturate at 2^64 - 1 in both, so they must be equal, on pairs whose band is
narrow (related), wide (one letter: the band hands the pair over), and absent (empty pairs),
around the edges of its 64-row and 64-column window.

The search appends runs of diagonal cells at once, keeps the lower stack entries and -- for
maps up to a limit, lowered here by PA_ENUM_MAP -- the current map in shared memory: its
results must be the host search's, result for result.
"""

import numpy as np
import pytest

from _cases import Gap
from test_gpu_enumerate import _compare_with_host, _solve, gpu_alg  # noqa: F401

pytestmark = pytest.mark.gpu


def _related(rng, n, letters, edits):
    a = rng.integers(0, letters, size=n).astype(np.uint32)
    b = list(a)
    for _ in range(edits):
        k = int(rng.integers(0, max(len(b), 1)))
        op = int(rng.integers(0, 3))
        if op == 0 and b:
            del b[min(k, len(b) - 1)]
        elif op == 1:
            b.insert(k, int(rng.integers(0, letters)))
        elif b:
            b[min(k, len(b) - 1)] = int(rng.integers(0, letters))
    return a, np.array(b, np.uint32)


def _long_pairs(rng, letters):
    pairs = [_related(rng, n, letters, 1 + n // 12) for n in (1, 7, 8, 9, 63, 64, 65, 255, 256, 257, 300, 521, 777)]
    pairs += [(rng.integers(0, letters, size=m).astype(np.uint32), rng.integers(0, letters, size=n).astype(np.uint32))
              for m, n in ((300, 40), (40, 300), (513, 600), (1, 400), (400, 1))]
    pairs.append((np.zeros(270, np.uint32), np.zeros(310, np.uint32)))  # every placement of the gap
    pairs.append((np.zeros(0, np.uint32), np.zeros(9, np.uint32)))
    pairs.append((np.zeros(300, np.uint32), np.zeros(0, np.uint32)))
    return pairs


@pytest.mark.parametrize("letters", [2, 4])
@pytest.mark.parametrize("locality", ["global", "semiglobal"])
@pytest.mark.parametrize("gap", ["linear", "affine", "free"])
@pytest.mark.parametrize("mode", ["G8", "chained", "chained8"])  # stripes of 128 and of 256 rows
def test_band_counts_equal_whole_matrix_counts(monkeypatch, gpu_alg, letters, locality, gap, mode):  # noqa: F811
    if mode.startswith("chained"):
        monkeypatch.setenv("PA_DP_MODE", "units")
        monkeypatch.setenv("PA_DP_ROWS", mode[7:] or "4")
    else:
        monkeypatch.setenv("PA_GROUP_WIDTH", mode[1:])
    pairs = _long_pairs(np.random.default_rng(77 + letters), letters)
    table = (3.0 * np.eye(letters) - 1.0).astype(np.float32)
    g = {"linear": Gap("linear", 1.0), "affine": Gap("affine", 2.0, 1.0), "free": Gap("affine", 0.0, 0.0)}[gap]
    got = {}
    for how in ("group", "chain", None):
        if how:
            monkeypatch.setenv("PA_COUNT_MODE", how)
        else:
            monkeypatch.delenv("PA_COUNT_MODE", raising=False)
        _, its, _, _, _, _ = _solve(gpu_alg, pairs, locality, g, "maximize", False, table)
        got[how] = [it.path_count() for it in its]
    assert got[None] == got["group"]
    assert got["chain"] == got["group"]


@pytest.mark.parametrize("locality", ["global", "semiglobal", "local"])
@pytest.mark.parametrize("gap", ["linear", "affine"])
@pytest.mark.parametrize("remove_dup", [True, False])
@pytest.mark.parametrize("most", ["", "64"])
def test_long_searches_match_host_search(monkeypatch, gpu_alg, locality, gap, remove_dup, most):  # noqa: F811
    if most:
        monkeypatch.setenv("PA_ENUM_MAP", most)
    monkeypatch.setenv("PA_GROUP_WIDTH", "8")
    pairs = _long_pairs(np.random.default_rng(5), 2)
    table = np.array([[2.0, -1.0], [-1.0, 2.0]], np.float32)
    g = Gap("linear", 1.0) if gap == "linear" else Gap("affine", 2.0, 1.0)
    _, its, ln, _, _, _ = _solve(gpu_alg, pairs, locality, g, "maximize", remove_dup, table)
    _compare_with_host(gpu_alg, its, ln, 40)
