"""Uneven pairs whose first tasks are spread over SMs and schedulers (needs a GPU): the same results
as from one counter (PA_GRID=exact) around the number of tasks where the spreading begins and past
its classes, and no slower than that."""

import ctypes

import numpy as np
import pytest

from _cases import Gap, options, pack, random_pairs

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def plan(monkeypatch):
    monkeypatch.setenv("PA_TUNE", "0")
    monkeypatch.setenv("PA_GROUP_WIDTH", "32")
    monkeypatch.setenv("PA_DP_MODE", "groups")
    monkeypatch.setenv("PA_DP16", "0")


def _solver(alg, n, lo, hi, gap):
    rng = np.random.default_rng(n)
    pairs = random_pairs(rng, n, lo, hi, alphabet=20)
    a, b, ln = pack(pairs, n)
    s = alg.m16.create_solver(a.shape[1], b.shape[1], alg.m16.create_options(
        options(alg, gap=gap, batch_size=n)))
    return s, lambda: s.solve_binary_for_alignment(a, b, 2.0, -1.0, ln)


@pytest.mark.parametrize("n", [600, 608, 609, 620, 1500, 2600])
@pytest.mark.parametrize("gap", [Gap("linear", 1.0), Gap("affine", 3.0, 1.0)])
def test_same_results(monkeypatch, n, gap):
    from pyalign_gb300 import algorithm as alg
    _, solve = _solver(alg, n, 40 if n > 1000 else 150, 400 if n > 1000 else 500, gap)
    got = solve()
    monkeypatch.setenv("PA_GRID", "exact")
    _, solve = _solver(alg, n, 40 if n > 1000 else 150, 400 if n > 1000 else 500, gap)
    for x, y in zip(got, solve()):
        assert x.score == y.score and np.array_equal(x.s_to_t, y.s_to_t)


@pytest.mark.parametrize("n", [590, 1000])
def test_not_slower_than_one_counter(monkeypatch, n):
    """The sweep's device time, best of 20; classes that ignored the schedulers took 1.2 to 1.4 times
    as long as the counter."""
    from pyalign_gb300 import algorithm as alg
    best = {}
    for grid in ("spread", "exact"):
        monkeypatch.setenv("PA_GRID", grid)
        s, solve = _solver(alg, n, 250, 500, Gap("affine", 3.0, 1.0))
        ms, launches, times = (ctypes.c_float * 4)(), ctypes.c_int32(), []
        for _ in range(20):
            solve()
            alg.lib().pa_solver_last_timings(s.handle, ms, ctypes.byref(launches))
            times.append(ms[1])
        best[grid] = min(times)
    assert best["spread"] <= 1.08 * best["exact"], best
