"""Alignments in untagged-range 16-bit twins (dps16_kernel with a traceback) against the int32
kernels and the oracle (needs a GPU).

The 16-bit launch must give the same scores and alignments as int32 (PA_DP16=0), whole numbers
both: pairs around the edges of 8-row lanes, stripes of every group width and 32-column chunks,
twins of unequal shape, empty pairs, an odd number of pairs, tie-rich and continuous-looking
tables, every locality, linear and affine gaps; values at the edge of the range (the launch must
then fall back or still be exact).
"""

import numpy as np
import pytest

from _cases import Gap, options, pack

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu_alg():
    from pyalign_gb300 import build
    build.build()
    from pyalign_gb300 import algorithm as alg
    if alg.lib().pa_device_count() == 0:
        pytest.fail("no CUDA device visible")
    return alg


def _pairs(rng, letters, sizes):
    pairs = []
    for n in sizes:
        a = rng.integers(0, letters, n).astype(np.uint32)
        b = a[rng.random(n) > 0.1].copy()
        hit = rng.random(len(b)) < 0.2
        b[hit] = rng.integers(0, letters, int(hit.sum()))
        pairs += [(a, b), (b, a), (a, rng.integers(0, letters, int(rng.integers(1, max(sizes) + 1))).astype(np.uint32))]
    pairs += [(pairs[0][0][:0], pairs[3][1]), (pairs[3][0], pairs[0][1][:0]), (np.zeros(0, np.uint32), np.zeros(0, np.uint32)),
              (np.zeros(40, np.uint32), np.full(50, letters - 1, np.uint32)),  # no match: a local optimum of 0
              (np.zeros(70, np.uint32), np.zeros(66, np.uint32))]
    order = rng.permutation(len(pairs))
    return [pairs[k] for k in order][: len(pairs) - 1 + len(pairs) % 2]


def _table(rng, letters, kind):
    if kind == "ties":
        return (2.0 * np.eye(letters) - 1.0).astype(np.float32)
    t = rng.integers(-6, 5, (letters, letters))
    t = np.minimum(t, t.T) + np.diag(rng.integers(4, 12, letters) + 6)
    return np.clip(t, -8, 14).astype(np.float32)


def _solve(alg, pairs, locality, gap, table):
    n = len(pairs)
    a, b, ln = pack(pairs, n)
    o = dict(options(alg, locality=locality, gap=gap), batch_size=n, batch=True)
    s = alg.m16.create_solver(a.shape[1], b.shape[1], alg.m16.create_options(o))
    return s, s.solve_indexed_for_alignment(a, b, table, ln)


def _same(got, want, what):
    assert len(got) == len(want)
    for k, (x, y) in enumerate(zip(got, want)):
        assert x.score == y.score, (what, k, x.score, y.score)
        assert np.array_equal(np.asarray(x.s_to_t), np.asarray(y.s_to_t)), (what, k)
        assert np.array_equal(np.asarray(x.t_to_s), np.asarray(y.t_to_s)), (what, k)


@pytest.mark.parametrize("locality", ["local", "global", "semiglobal"])
@pytest.mark.parametrize("gap", ["linear", "affine"])
@pytest.mark.parametrize("letters,kind", [(3, "ties"), (20, "ties"), (20, "scores"), (32, "scores")])
@pytest.mark.parametrize("mode", ["G1", "G4", "G8", "G32", "chained"])
def test_alignments_equal_int32(monkeypatch, gpu_alg, locality, gap, letters, kind, mode):
    if mode == "chained":
        monkeypatch.setenv("PA_DP_MODE", "units")
    else:
        monkeypatch.setenv("PA_GROUP_WIDTH", mode[1:])
    monkeypatch.setenv("PA_DP16", "all")
    rng = np.random.default_rng(letters + len(mode))
    sizes = (1, 2, 7, 8, 9, 31, 33, 64, 65) if mode == "G1" else (1, 8, 9, 31, 32, 33, 63, 65, 129, 255, 256, 257, 300, 530)
    pairs = _pairs(rng, letters, sizes)
    table = _table(rng, letters, kind)
    g = Gap("linear", 2.0) if gap == "linear" else Gap("affine", 3.0, 1.0)
    s, got = _solve(gpu_alg, pairs, locality, g, table)
    if letters > 4 or locality == "semiglobal":
        assert s.last_plan()["arithmetic"] == "int16x2", s.last_plan()
    monkeypatch.setenv("PA_DP16", "0")
    s, want = _solve(gpu_alg, pairs, locality, g, table)
    assert s.last_plan()["arithmetic"] == "int32", s.last_plan()
    _same(got, want, (locality, gap, mode))


@pytest.mark.parametrize("locality", ["local", "global", "semiglobal"])
@pytest.mark.parametrize("gap", ["linear", "affine"])
def test_alignments_equal_the_oracle(monkeypatch, gpu_alg, oracle_alg, locality, gap):
    monkeypatch.setenv("PA_GROUP_WIDTH", "8")
    monkeypatch.setenv("PA_DP16", "all")
    rng = np.random.default_rng(4)
    pairs = _pairs(rng, 20, (1, 5, 8, 17, 32, 40, 70))
    table = _table(rng, 20, "scores")
    g = Gap("linear", 2.0) if gap == "linear" else Gap("affine", 3.0, 1.0)
    s, got = _solve(gpu_alg, pairs, locality, g, table)
    assert s.last_plan()["arithmetic"] == "int16x2", s.last_plan()
    _same(got, _solve(oracle_alg, pairs, locality, g, table)[1], (locality, gap))


@pytest.mark.parametrize("locality", ["local", "global", "semiglobal"])
@pytest.mark.parametrize("top", [7, 13, 26, 28])
def test_values_around_the_edge_of_the_range(monkeypatch, gpu_alg, locality, top):
    """top * 300 quadrupled: 8,400 .. 33,600, below and past 16 bits."""
    monkeypatch.setenv("PA_GROUP_WIDTH", "16")
    monkeypatch.setenv("PA_DP16", "all")
    rng = np.random.default_rng(top)
    pairs = [(a := rng.integers(0, 20, 300).astype(np.uint32), a.copy()) for _ in range(5)]
    pairs += _pairs(rng, 20, (30, 300))
    table = (float(top + 4) * np.eye(20) - 4.0).astype(np.float32)
    s, got = _solve(gpu_alg, pairs, locality, Gap("affine", 11.0, 1.0), table)
    monkeypatch.setenv("PA_DP16", "0")
    _same(got, _solve(gpu_alg, pairs, locality, Gap("affine", 11.0, 1.0), table)[1], (locality, top))


@pytest.mark.parametrize("locality", ["local", "global", "semiglobal"])
def test_repeated_host_calls_run_as_a_pipeline(monkeypatch, gpu_alg, locality):
    """8,401 short pairs: the second call on one solver runs in chunks on two streams."""
    monkeypatch.setenv("PA_TUNE", "0")
    rng = np.random.default_rng(12)
    n = 8401
    a, b = (rng.integers(0, 20, (n, 40)).astype(np.uint32) for _ in range(2))
    b[::2] = a[::2]
    b[:, 7::9] = rng.integers(0, 20, b[:, 7::9].shape)
    ln = rng.integers(1, 41, (2, n)).astype(np.uint16)
    table = _table(rng, 20, "scores")
    got = {}
    for dp16 in ("0", "all"):
        monkeypatch.setenv("PA_DP16", dp16)
        o = dict(options(gpu_alg, locality=locality, gap=Gap("affine", 5.0, 1.0)), batch_size=n, batch=True)
        s = gpu_alg.m16.create_solver(40, 40, gpu_alg.m16.create_options(o))
        got[dp16] = [[(x.score, np.asarray(x.s_to_t).tobytes(), np.asarray(x.t_to_s).tobytes())
                      for x in s.solve_indexed_for_alignment(a, b, table, ln)] for _ in range(3)]
        assert s.last_plan()["arithmetic"] == ("int32" if dp16 == "0" else "int16x2")
    for calls in got["all"] + got["0"][1:]:
        assert calls == got["0"][0]
