"""Scores alone in packed 16-bit twins against the oracle: stripe, row and column edges, alphabets
on both sides of its profiles, every locality, group width and mode, twins of unlike shapes, and
launches just inside and just outside its bounds (those run in int32, with the same scores)."""

import numpy as np
import pytest

from _cases import Gap, call, compare, options, pack, random_pairs

pytestmark = pytest.mark.gpu


def pairs_of(rng, letters, hi):
    edge = [(0, 9), (9, 0), (300, 0), (0, 300), (1, 1), (1, 2), (2, 1), (7, 8), (8, 7), (9, 15), (31, 32), (33, 31),
            (63, 64), (65, 33), (128, 127), (255, 257), (257, 255), (256, 64), (5, hi), (hi, 5), (hi, hi)]
    out = []
    for n, m in edge:
        s = rng.integers(0, letters, n).astype(np.uint32)
        t = np.resize(s, m) if n and rng.random() < 0.5 else rng.integers(0, letters, m)
        out.append((s, t.astype(np.uint32)))
    return out + random_pairs(rng, 20, 1, hi, alphabet=letters, related=0.6)


def check(gpu_alg, oracle_alg, pairs, table, locality, direction, gap, arithmetic="int16x2"):
    a, b, ln = pack(pairs, len(pairs))
    o = options(gpu_alg, locality=locality, direction=direction, detail="score", gap=gap, batch_size=len(pairs))
    args = (o, (a.shape[1], b.shape[1]), "score", "indexed", a, b, ln, table)
    solver, g = call(gpu_alg, *args)
    assert solver.last_plan()["arithmetic"] == arithmetic, solver.last_plan()
    d = compare("score", g, call(oracle_alg, *args)[1], len(pairs))
    assert d is None, d
    return solver.last_plan()


@pytest.mark.parametrize("mode", ["1", "2", "4", "8", "16", "32", "units"])
@pytest.mark.parametrize("locality", ["local", "global", "semiglobal"])
@pytest.mark.parametrize("letters", [2, 4, 5, 20, 32])
@pytest.mark.parametrize("gap", [Gap("linear", 2.0), Gap("affine", 7.0, 1.0), Gap("affine", 3.0, 0.0)])
def test_scores(monkeypatch, oracle_alg, mode, locality, letters, gap):
    from pyalign_gb300 import algorithm as gpu_alg
    monkeypatch.setenv("PA_TUNE", "0")
    if mode == "units":
        monkeypatch.setenv("PA_DP_MODE", "units")
    else:
        monkeypatch.setenv("PA_GROUP_WIDTH", mode)
    rng = np.random.default_rng(letters * 7 + len(locality))
    direction = "minimize" if letters == 5 else "maximize"
    table = rng.integers(-4, 3, size=(letters, letters)).astype(np.float32)
    np.fill_diagonal(table, rng.integers(4, 12, letters))
    plan = check(gpu_alg, oracle_alg, pairs_of(rng, letters, 320), table if direction == "maximize" else -table, locality,
                 direction, gap)
    assert plan["kernel"] == ("stripe-chained" if mode == "units" else "16-bit twins, two-column")


@pytest.mark.parametrize("locality,inside,outside", [
    # the largest similarity, so that its sum over 300 rows is just representable or just not
    ("local", 109, 110), ("semiglobal", 127, None), ("global", 127, None)])
def test_bounds(monkeypatch, oracle_alg, locality, inside, outside):
    from pyalign_gb300 import algorithm as gpu_alg
    monkeypatch.setenv("PA_TUNE", "0")
    monkeypatch.setenv("PA_DP_MODE", "groups")
    s = np.zeros(300, np.uint32)
    pairs = [(s, s), (s[:200], s), (s, s[:10]), (np.ones(300, np.uint32), s)]
    for top, arithmetic in ((inside, "int16x2"), (outside, "int32")):
        if top is None:
            continue
        table = np.array([[top, -128], [-100, 3]], np.float32)
        check(gpu_alg, oracle_alg, pairs, table, locality, "maximize", Gap("affine", 20.0, 10.0), arithmetic)
    # similarities past int8, a gap that pays
    check(gpu_alg, oracle_alg, pairs, np.array([[128, -1], [-1, 2]], np.float32), locality, "maximize", Gap("linear", 2.0),
          "int32")
    check(gpu_alg, oracle_alg, pairs, np.array([[2, -9], [-9, 2]], np.float32), locality, "maximize",
          Gap("linear", -1.0), "int32")


@pytest.mark.parametrize("locality", ["global", "semiglobal"])
def test_wide_range(monkeypatch, oracle_alg, locality):
    """Values over most of the 16-bit range: long gaps against long matches, chained and not."""
    from pyalign_gb300 import algorithm as gpu_alg
    monkeypatch.setenv("PA_TUNE", "0")
    rng = np.random.default_rng(8)
    s = rng.integers(0, 4, 2000).astype(np.uint32)
    pairs = [(s, s), (s[:1], s), (s, s[:1]), (s, s[::-1].copy()), (s[:700], s[300:])]
    table = np.full((4, 4), -5.0, np.float32)
    np.fill_diagonal(table, 11.0)
    for mode in ("units", "groups"):
        monkeypatch.setenv("PA_DP_MODE", mode)
        check(gpu_alg, oracle_alg, pairs, table, locality, "maximize", Gap("affine", 10.0, 4.0))
