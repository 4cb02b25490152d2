"""The two-column float kernel against the one-column kernel (PA_DP_COLS=1), bit for bit: scores and
paths at the edges of its stripes, rows and column pairs, over the layouts of a dense similarity
it reads in place or copies first, with cells of -inf, +inf and NaN, for series and for tables."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [(1, 1), (1, 9), (9, 1), (3, 2), (4, 5), (5, 4), (7, 8), (8, 7), (31, 33), (64, 63), (65, 128), (127, 129),
           (0, 4), (4, 0), (130, 2), (2, 130)]


def solve(monkeypatch, cols, G, fn):
    from pyalign_gb300 import autograd as ag
    if cols == 1:
        monkeypatch.setenv("PA_DP_COLS", "1")
    else:
        monkeypatch.delenv("PA_DP_COLS", raising=False)
    monkeypatch.setenv("PA_GROUP_WIDTH", str(G))
    ag._SOLVERS.clear()
    scores, paths, plen, poff = fn()[:4]
    plan = list(ag._SOLVERS.values())[0].last_plan()
    ag._SOLVERS.clear()
    s, p, n, o = (x.cpu().numpy() for x in (scores, paths, plen, poff))
    return s, [p[o[k]:o[k] + 2 * n[k]] for k in range(len(n))], plan["kernel"]


def same(x, y):
    assert np.array_equal(x[0], y[0], equal_nan=True)
    for a, b in zip(x[1], y[1]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("layout", ["transposed", "rows", "odd_pitch", "offset", "odd_rows"])
@pytest.mark.parametrize("locality,direction,gap", [
    ("local", "maximize", (0.5, 0.1)), ("global", "minimize", (0.75, 0.25)), ("semiglobal", "maximize", (0.5, 0.5)),
    ("local", "minimize", (0.3, None)), ("global", "maximize", (0.25, None)), ("semiglobal", "minimize", (0.5, None)),
    ("global", "minimize", None)])
@pytest.mark.parametrize("values", ["random", "ties", "special"])
def test_dense_layouts(monkeypatch, layout, locality, direction, gap, values):
    import torch
    from pyalign_gb300 import autograd as ag
    rng = np.random.default_rng(len(layout) * 100 + len(locality) * 10 + len(values))
    B, n, m = len(LENGTHS), 130 + (2 if layout != "odd_rows" else 1), 130
    S = rng.random((B, n, m)).astype(np.float32) * 2 - 1
    if values == "ties":
        S = np.round(S * 2) / 4
    if values == "special":
        S[rng.random(S.shape) < 0.2] = -np.inf if direction == "maximize" else np.inf
        S[rng.random(S.shape) < 0.002] = np.nan
        S[rng.random(S.shape) < 0.001] = np.inf if direction == "maximize" else -np.inf
    x = torch.from_numpy(S.astype(np.float32)).cuda()
    if layout == "transposed" or layout == "odd_rows":
        x = x.transpose(1, 2).contiguous().transpose(1, 2)
    elif layout == "odd_pitch":
        x = torch.nn.functional.pad(x.transpose(1, 2), (0, 3)).contiguous()[:, :, :n].transpose(1, 2)
    elif layout == "offset":
        big = torch.zeros(B, m, n + 8, device="cuda")
        big[:, :, 1:n + 1] = x.transpose(1, 2)
        x = big[:, :, 1:n + 1].transpose(1, 2)

    def fn():
        return ag._forward_paths(x, np.array(LENGTHS), None if gap is None else gap, locality, direction, gap is None)
    for G in (1, 4, 8, 32):
        one, two = solve(monkeypatch, 1, G, fn), solve(monkeypatch, 2, G, fn)
        assert one[2] == "one-column" and two[2] == "two-column"
        same(one, two)


@pytest.mark.parametrize("dtw", [True, False])
def test_series(monkeypatch, dtw):
    import torch
    from pyalign_gb300 import autograd as ag
    rng = np.random.default_rng(3)
    x, y = (torch.from_numpy(np.round(rng.random((len(LENGTHS), 130)) * 8).astype(np.float32) / 4).cuda() for _ in range(2))
    for G in (1, 4, 16, 32):
        def fn():
            return ag._series_paths(x, y, np.array(LENGTHS), None if dtw else (0.5, 0.25), "global", "minimize", dtw)
        same(solve(monkeypatch, 1, G, fn), solve(monkeypatch, 2, G, fn))


@pytest.mark.parametrize("locality", ["local", "global", "semiglobal"])
@pytest.mark.parametrize("letters", [4, 20, 90])
@pytest.mark.parametrize("gap", [("linear", 0.5), ("affine", 1.5, 0.25)])
def test_table(monkeypatch, oracle_alg, locality, letters, gap):
    """Tables in shared memory and past its 64 x 64 limit, scores alone and alignments, against
    the oracle."""
    from _cases import Gap, call, compare, options, pack, random_pairs
    from pyalign_gb300 import algorithm as gpu_alg
    rng = np.random.default_rng(letters + len(locality))
    pairs = random_pairs(rng, 24, 1, 140, alphabet=letters)
    a, b, ln = pack(pairs, len(pairs))
    table = (rng.random((letters, letters)) * 3 - 1.5).astype(np.float32)
    np.fill_diagonal(table, 2.25)
    for G in (1, 8, 32):
        monkeypatch.setenv("PA_GROUP_WIDTH", str(G))
        for method in ("score", "alignment"):
            o = options(gpu_alg, locality=locality, detail=method, gap=Gap(*gap), batch_size=len(pairs))
            args = (o, (a.shape[1], b.shape[1]), method, "indexed", a, b, ln, table)
            solver, g = call(gpu_alg, *args)
            assert solver.last_plan()["kernel"] == "two-column" and solver.last_plan()["arithmetic"] == "float32"
            assert compare(method, g, call(oracle_alg, *args)[1], len(pairs)) is None
