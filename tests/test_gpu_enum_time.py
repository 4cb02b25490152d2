"""The device enumeration in bounded launches (needs a GPU): a search that pauses and goes on gives the
same results as one that does not, and pairs whose co-optimal paths are beyond counting but spell
one alignment come back cut off instead of holding the GPU."""

import time

import numpy as np
import pytest

from _cases import Gap, options, pack, random_pairs

pytestmark = pytest.mark.gpu


def _iterators(alg, pairs, locality, gap, dup=False):
    a, b, ln = pack(pairs, len(pairs))
    o = options(alg, locality=locality, gap=gap, count="all", batch_size=len(pairs), return_dup=dup)
    s = alg.m16.create_solver(a.shape[1], b.shape[1], alg.m16.create_options(o))
    return s, s.solve_binary_for_alignment_iterator(a, b, 1.0, -1.0, ln)


@pytest.mark.parametrize("locality", ["local", "global", "semiglobal"])
@pytest.mark.parametrize("gap", [Gap("linear", 1.0), Gap("affine", 2.0, 1.0)])
@pytest.mark.parametrize("dup", [False, True])
@pytest.mark.parametrize("env", [{}, {"PA_ENUM_MAP": "0"}, {"PA_ENUM_STACK": "3"}])
def test_pauses_change_nothing(monkeypatch, locality, gap, dup, env):
    from pyalign_gb300 import algorithm as alg
    rng = np.random.default_rng(5)
    pairs = random_pairs(rng, 12, 1, 24, alphabet=4) + random_pairs(rng, 2, 300, 400, alphabet=20, related=1.0)
    _, its = _iterators(alg, pairs, locality, gap, dup)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    want = alg.FirstAlignments(its[0]._res, 12, with_paths=True)
    monkeypatch.setenv("PA_ENUM_CYCLES", "0")  # pauses at every duplicate
    got = alg.FirstAlignments(its[0]._res, 12, with_paths=True)
    assert not want.more.any() and not got.more.any()
    for name in ("counts", "maps", "paths", "plen"):
        x, y = getattr(got, name), getattr(want, name)
        if name == "paths":  # only the points of each result's walk are written
            for lane in range(len(pairs)):
                for j in range(int(want.counts[lane])):
                    assert np.array_equal(got.alignment(lane, j)[1], want.alignment(lane, j)[1])
        else:
            assert np.array_equal(x, y), name


def test_uncountable_paths_of_one_alignment(monkeypatch):
    """30 letters against 30 others without gap costs: C(60, 30) paths, all of them the empty map."""
    from pyalign_gb300 import algorithm as alg
    monkeypatch.setattr(alg.FirstAlignments, "SECONDS", 0.2)
    few = (np.arange(4, dtype=np.uint32), np.arange(4, dtype=np.uint32))
    pairs = [(np.zeros(30, np.uint32), np.ones(30, np.uint32)), few]
    _, its = _iterators(alg, pairs, "global", Gap("linear", 0.0))
    begun = time.time()
    first = its[0].next()
    assert time.time() - begun < 10
    assert first.score == 0 and (np.asarray(first.s_to_t) == -1).all()
    f = its[0]._res._first[False]
    assert f.counts[0] == 1 and f.more[0] == 1
    assert f.more[1] == 0 and np.array_equal(its[1].next().s_to_t, np.arange(4))
