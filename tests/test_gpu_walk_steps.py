"""The traceback walk step by step against the oracle and against the path's own cost (needs a GPU).

Where diagonal runs are short, linear-gap and DTW paths are walked 32 steps at a time inside the
32 x 32 window of traceback words; pairs here cross its edges, switch between runs and steps
(related pairs with unrelated stretches), and end on every border.  Alignments are whole numbers
and must equal the oracle's.  DTW series hold small integers, so costs are exact.
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


@pytest.mark.parametrize("locality", ["local", "global", "semiglobal"])
@pytest.mark.parametrize("width", ["4", "32", None])
@pytest.mark.parametrize("scores", ["whole", "fraction"])
def test_linear_alignments_equal_the_oracle(monkeypatch, gpu_alg, oracle_alg, locality, width, scores):
    if width:
        monkeypatch.setenv("PA_GROUP_WIDTH", width)
    rng = np.random.default_rng(8)
    pairs = []
    for n in (1, 2, 7, 8, 9, 31, 32, 33, 63, 64, 65, 96, 130):
        a = rng.integers(0, 4, n).astype(np.uint32)
        b = a.copy()
        b[n // 3:2 * n // 3] = rng.integers(0, 4, 2 * n // 3 - n // 3)  # a related pair with an unrelated middle
        pairs += [(a, b), (a, rng.integers(0, 4, int(rng.integers(1, 131))).astype(np.uint32)),
                  (a[: max(1, n // 4)], b), (a, np.roll(b, n // 2))]
    n = len(pairs)
    a, b, ln = pack(pairs, n)
    f = 1.0 if scores == "whole" else 0.5
    table = (f * (3.0 * np.eye(4) - 1.0)).astype(np.float32)
    o = dict(options(gpu_alg, locality=locality, gap=Gap("linear", f)), batch_size=n, batch=True)
    cap = (a.shape[1], b.shape[1])
    got = gpu_alg.m16.create_solver(*cap, gpu_alg.m16.create_options(o)).solve_indexed_for_alignment(a, b, table, ln)
    want = oracle_alg.m16.create_solver(*cap, oracle_alg.m16.create_options(o)).solve_indexed_for_alignment(a, b, table, ln)
    for k in range(n):
        assert got[k].score == want[k].score, k
        assert np.array_equal(np.asarray(got[k].s_to_t), np.asarray(want[k].s_to_t)), k
        assert np.array_equal(np.asarray(got[k].t_to_s), np.asarray(want[k].t_to_s)), k


def test_dtw_paths_cost_their_scores(gpu_alg):
    torch = pytest.importorskip("torch")
    from pyalign_gb300 import autograd as ag
    rng = np.random.default_rng(9)
    lengths = np.array([[1, 1], [1, 40], [40, 1], [31, 32], [32, 33], [33, 31], [64, 65], [100, 7], [200, 190], [190, 200],
                        [200, 200], [65, 128]])
    B, n = len(lengths), 200
    x, y = (np.cumsum(rng.integers(-3, 4, (B, n)), 1).astype(np.float32) for _ in range(2))
    y[10] = x[10]  # all diagonal
    X, Y = torch.tensor(x, device="cuda"), torch.tensor(y, device="cuda")
    scores, paths, plen, poff = ag._series_paths(X, Y, lengths, None, "global", "minimize", True)
    paths, plen, poff = paths.cpu().numpy(), plen.cpu().numpy(), poff.cpu().numpy()
    for k, (ls, lt) in enumerate(lengths):
        D = np.full((ls + 1, lt + 1), np.inf)
        D[0, 0] = 0.0
        for i in range(ls):
            for j in range(lt):
                D[i + 1, j + 1] = abs(x[k, i] - y[k, j]) + min(D[i, j], D[i, j + 1], D[i + 1, j])
        P = paths[poff[k]:poff[k] + 2 * plen[k]].reshape(-1, 2)
        assert float(scores[k]) == D[ls, lt], k
        assert tuple(P[0]) == (ls - 1, lt - 1), k
        step = P[:-1] - P[1:]
        assert ((step >= 0) & (step <= 1)).all() and (step.sum(1) >= 1).all(), k
        inside = P[(P >= 0).all(1)]
        assert tuple(inside[-1]) == (0, 0) or (inside[-1] == 0).any(), k
        cost = sum(abs(float(x[k, u]) - float(y[k, v])) for u, v in inside)
        u, v = inside[-1]  # a path that leaves along a border pays its remaining cells
        cost += sum(abs(float(x[k, i]) - float(y[k, 0])) for i in range(u)) if v == 0 else 0.0
        cost += sum(abs(float(x[k, 0]) - float(y[k, j])) for j in range(v)) if u == 0 else 0.0
        assert cost == D[ls, lt], k
