"""Which arithmetic alignments run in around the edge of the 16-bit twins' range, and that the results
there are the oracle's (needs a GPU).

Values are held times 4 plus a tag.  Local alignment uses the upper half of 16 bits: 300 matches of 27
reach 32,400 + 3 <= 32,767, of 28 they do not.  Global and semiglobal alignment use the whole range, of
which 300 matches take less than the largest similarity allowed, 31 (31 * 4 + 2 is the last below
128)."""

import numpy as np
import pytest

from _cases import Gap, options, pack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("locality,top,arithmetic", [
    ("local", 26, "int16x2"), ("local", 27, "int16x2"), ("local", 28, "int32"), ("local", 31, "int32"),
    ("global", 28, "int16x2"), ("global", 31, "int16x2"), ("global", 32, "int32"),
    ("semiglobal", 28, "int16x2"), ("semiglobal", 31, "int16x2"), ("semiglobal", 32, "int32")])
@pytest.mark.parametrize("mode", ["16", "units"])
def test_arithmetic_and_results(monkeypatch, oracle_alg, locality, top, arithmetic, mode):
    from pyalign_gb300 import algorithm as gpu_alg
    if mode == "units":
        monkeypatch.setenv("PA_DP_MODE", "units")
    else:
        monkeypatch.setenv("PA_GROUP_WIDTH", mode)
    monkeypatch.setenv("PA_DP16", "all")
    rng = np.random.default_rng(top)
    pairs = [(a := rng.integers(0, 20, 300).astype(np.uint32), a.copy()) for _ in range(3)]  # the largest value
    pairs += [(np.zeros(300, np.uint32), np.ones(300, np.uint32)),                           # the smallest
              (pairs[0][0][:40], pairs[0][0]), (pairs[1][0], pairs[1][0][100:])]
    a, b, ln = pack(pairs, len(pairs))
    table = (float(top + 4) * np.eye(20) - 4.0).astype(np.float32)

    def solve(alg):
        o = options(alg, locality=locality, gap=Gap("affine", 11.0, 1.0), batch_size=len(pairs))
        s = alg.m16.create_solver(300, 300, alg.m16.create_options(o))
        return s, s.solve_indexed_for_alignment(a, b, table, ln)

    solver, got = solve(gpu_alg)
    assert solver.last_plan()["arithmetic"] == arithmetic, solver.last_plan()
    for x, y in zip(got, solve(oracle_alg)[1]):
        assert x.score == y.score
        assert np.array_equal(np.asarray(x.s_to_t), np.asarray(y.s_to_t))
