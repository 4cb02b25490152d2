"""Two threads with a solver each, whose launches of one kernel ask for different amounts of shared
memory above the default limit (needs a GPU): every solve succeeds and gives the same result."""

import threading

import numpy as np
import pytest

from _cases import Gap, options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("detail", ["score", "alignment"])
def test_alphabets_of_24_and_32_letters(monkeypatch, detail):
    from pyalign_gb300 import algorithm as alg
    monkeypatch.setenv("PA_TUNE", "0")
    monkeypatch.setenv("PA_GROUP_WIDTH", "8")
    monkeypatch.setenv("PA_DP16", "all")
    n, size, calls = 64, 40, 10000
    errors = []
    start = threading.Barrier(2)

    def work(letters):
        try:
            rng = np.random.default_rng(letters)
            a, b = (rng.integers(0, letters, (n, size)).astype(np.uint32) for _ in range(2))
            table = (6.0 * np.eye(letters) - 2.0).astype(np.float32)
            length = np.full((2, n), size, np.uint16)
            o = options(alg, locality="global", gap=Gap("affine", 3.0, 1.0), detail=detail, batch_size=n)
            solver = alg.m16.create_solver(size, size, alg.m16.create_options(o))
            if detail == "score":
                solve = lambda: solver.solve_indexed_for_score(a, b, table, length)  # noqa: E731
            else:
                solve = lambda: [x.score for x in solver.solve_indexed_for_alignment(a, b, table, length)]  # noqa: E731
            start.wait(60)
            want = np.array(solve())
            for k in range(calls if detail == "score" else calls // 8):
                assert np.array_equal(np.array(solve()), want), k
            assert solver.last_plan()["arithmetic"] == "int16x2", solver.last_plan()
        except BaseException as e:  # noqa: BLE001
            errors.append((letters, repr(e)))

    threads = [threading.Thread(target=work, args=(letters,)) for letters in (24, 32)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
