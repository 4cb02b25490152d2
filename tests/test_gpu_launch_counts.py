"""The reported kernel launches of a solve (needs a GPU): in one piece and as a pipeline of chunks,
one code check for both sequences, one sweep and one walk each."""

import ctypes

import numpy as np
import pytest

from _cases import Gap, options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunks", [1, 2, 3])
@pytest.mark.parametrize("form", ["indexed", "binary"])
def test_launches_of_a_repeated_host_solve(monkeypatch, chunks, form):
    from pyalign_gb300 import algorithm as alg
    monkeypatch.setenv("PA_CHUNKS", str(chunks))
    monkeypatch.setenv("PA_TUNE", "0")
    monkeypatch.setenv("PA_DP_MODE", "groups")
    rng = np.random.default_rng(3)
    a, b = (rng.integers(0, 4, (64, 30)).astype(np.uint32) for _ in range(2))
    ln = np.full((2, 64), 30, np.uint16)
    s = alg.m16.create_solver(30, 30, alg.m16.create_options(options(alg, gap=Gap("linear", 1.0), batch_size=64)))
    ms, launches = (ctypes.c_float * 4)(), ctypes.c_int32()
    for call in range(3):
        if form == "indexed":
            s.solve_indexed_for_alignment(a, b, (2.0 * np.eye(4) - 1.0).astype(np.float32), ln)
        else:
            s.solve_binary_for_alignment(a, b, 1.0, -1.0, ln)
        alg.lib().pa_solver_last_timings(s.handle, ms, ctypes.byref(launches))
        pieces = 1 if call == 0 else chunks  # the first call runs in one piece of work per kernel
        want = (3 if form == "indexed" else 2) * pieces
        assert launches.value == want, (call, launches.value, want)
