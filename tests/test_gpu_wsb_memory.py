"""General gap costs of narrow pairs with little memory free (needs a GPU): the tiled sweep's whole
tiles do not fit, the cells do, and the solve gives the same alignments."""

import numpy as np
import pytest

from _cases import Gap, options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("detail", ["alignment", "score"])
def test_one_row_against_many_columns(detail):
    import torch

    from pyalign_gb300 import algorithm as alg
    rng = np.random.default_rng(1)
    n, m = 3000, 3000  # 9 M cells, in whole tiles 2 x 1.15 GB
    a, b = rng.integers(0, 4, (n, 1)).astype(np.uint32), rng.integers(0, 4, (n, m)).astype(np.uint32)
    ln = np.stack([np.ones(n), rng.integers(m - 20, m + 1, n)]).astype(np.uint16)
    table = (3.0 * np.eye(4) - 1.0).astype(np.float32)

    def solve():
        s = alg.m16.create_solver(1, m, alg.m16.create_options(
            options(alg, locality="global", gap=Gap("log", 1.0, 0.5), detail=detail, batch_size=n)))
        if detail == "score":
            return np.asarray(s.solve_indexed_for_score(a, b, table, ln))
        return [(x.score, x.s_to_t.tobytes()) for x in s.solve_indexed_for_alignment(a, b, table, ln)]

    want = solve()
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (1 << 30), dtype=torch.uint8, device="cuda")
    try:
        got = solve()
    finally:
        del fill
        torch.cuda.empty_cache()
    assert np.array_equal(got, want) if detail == "score" else got == want
