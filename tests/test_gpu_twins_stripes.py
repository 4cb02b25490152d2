"""16-bit twins whose two pairs have different numbers of 256-row stripes (needs a GPU): every
class of stripes holds an odd number of pairs, so the processing order pairs the last of one class
with the first of the next, and the shorter pair's last row lies in an earlier stripe than the
twin's last.

Semiglobal optima of the pairs lie in the last row away from its end, strictly better than the last
column or equal to it (the last row then goes first), and in the last column; compared with the
oracle and with the int32 kernels, whole numbers both."""

import numpy as np
import pytest

from _cases import Gap, options, pack

pytestmark = pytest.mark.gpu

SHAPES = [(600, 300), (600, 300, 100), (600, 300, 300, 100, 40), (300, 100), (300, 0, 100), (600, 100, 520, 30, 257),
          (1000, 300, 600, 100, 90)]


def _pair(rng, letters, n, kind):
    """A sequence of n letters and one that puts the optimum where `kind` says.  The filler avoids
    the sequence's own letters as far as the alphabet allows."""
    s = rng.integers(0, letters - 1, n).astype(np.uint32)
    filler = np.full(60, letters - 1, np.uint32)
    h = n // 2
    if kind == "row":       # all of s inside t: it ends in the last row
        t = np.concatenate([filler, s, filler])
    elif kind == "column":  # t inside s: it ends in the last column
        t = s[n // 4: n // 4 + h]
    else:                   # s = P + Q, t = Q + filler + P: Q ends in the last row, P in the last column
        t = np.concatenate([s[h:2 * h], filler, s[:h]])
    return (s[:2 * h] if kind == "tie" else s), t.astype(np.uint32)


def _solve(alg, pairs, locality, gap, table, detail="alignment"):
    a, b, ln = pack(pairs, len(pairs))
    o = options(alg, locality=locality, gap=gap, detail=detail, batch_size=len(pairs))
    s = alg.m16.create_solver(a.shape[1], b.shape[1], alg.m16.create_options(o))
    if detail == "score":
        return s, np.asarray(s.solve_indexed_for_score(a, b, table, ln))
    return s, s.solve_indexed_for_alignment(a, b, table, ln)


@pytest.fixture(scope="module")
def gpu_alg():
    from pyalign_gb300 import build
    build.build()
    from pyalign_gb300 import algorithm as alg
    if alg.lib().pa_device_count() == 0:
        pytest.fail("no CUDA device visible")
    return alg


@pytest.mark.parametrize("mode", ["chained", "G32", "G8"])
@pytest.mark.parametrize("kind", ["row", "tie", "column"])
@pytest.mark.parametrize("locality", ["semiglobal", "global", "local"])
@pytest.mark.parametrize("letters", [4, 20])
@pytest.mark.parametrize("gap", ["linear", "affine"])
def test_stripe_classes_of_odd_size(monkeypatch, gpu_alg, oracle_alg, mode, kind, locality, letters, gap):
    monkeypatch.setenv("PA_TUNE", "0")
    if mode == "chained":
        monkeypatch.setenv("PA_DP_MODE", "units")
    else:
        monkeypatch.setenv("PA_GROUP_WIDTH", mode[1:])
    rng = np.random.default_rng(letters)
    table = (8.0 * np.eye(letters) - 5.0).astype(np.float32)
    g = Gap("linear", 3.0) if gap == "linear" else Gap("affine", 6.0, 2.0)
    for shape in SHAPES:
        pairs = [_pair(rng, letters, n, kind) for n in shape]
        want = _solve(oracle_alg, pairs, locality, g, table)[1]
        if locality == "semiglobal" and kind != "column":
            for (s, t), w in zip(pairs, want):  # the optimum is in the last row, not at its end
                assert len(s) == 0 or 0 <= np.asarray(w.s_to_t)[-1] < len(t) - 1
        for dp16, arithmetic in (("all", "int16x2"), ("0", "int32")):
            monkeypatch.setenv("PA_DP16", dp16)
            solver, got = _solve(gpu_alg, pairs, locality, g, table)
            assert solver.last_plan()["arithmetic"] == arithmetic, (shape, solver.last_plan())
            for k, (x, y) in enumerate(zip(got, want)):
                assert x.score == y.score, (dp16, shape, k, x.score, y.score)
                assert np.array_equal(np.asarray(x.s_to_t), np.asarray(y.s_to_t)), (dp16, shape, k)
            scores = _solve(gpu_alg, pairs, locality, g, table, "score")[1]
            assert np.array_equal(scores, np.array([y.score for y in want], np.float32)), (dp16, shape)
