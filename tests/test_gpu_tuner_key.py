"""Launches that choose between different kernels do not share a measured plan (needs a GPU): after a
launch was tuned, one of the same sizes that other kernels may take is tuned on its own, and one
more of the same kind takes its plan over.  A tuning call is told by its many kernel launches."""

import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

RUN = r"""
import ctypes, json, sys
sys.path[:0] = sys.argv[1:3]
import numpy as np
from _cases import Gap, options
from pyalign_gb300 import algorithm as alg

def launches(solver):
    ms, n = (ctypes.c_float * 4)(), ctypes.c_int32()
    alg.lib().pa_solver_last_timings(solver.handle, ms, ctypes.byref(n))
    return n.value

def indexed(letters):
    rng = np.random.default_rng(letters)
    a, b = (rng.integers(0, letters, (1100, 64)).astype(np.uint32) for _ in range(2))
    ln = np.full((2, 1100), 64, np.uint16)
    s = alg.m16.create_solver(64, 64, alg.m16.create_options(
        options(alg, gap=Gap("affine", 3.0, 1.0), detail="score", batch_size=1100)))
    s.solve_indexed_for_score(a, b, (4.0 * np.eye(letters) - 2.0).astype(np.float32), ln)
    return launches(s)

def aligned(locality):
    rng = np.random.default_rng(1)
    a, b = (rng.integers(0, 5, (2100, 380)).astype(np.uint32) for _ in range(2))
    s = alg.m16.create_solver(380, 380, alg.m16.create_options(
        options(alg, gap=Gap("linear", 2.0), locality=locality, batch_size=2100)))
    s.solve_indexed_for_alignment(a, b, (4.0 * np.eye(5) - 2.0).astype(np.float32), np.full((2, 2100), 380, np.uint16))
    return launches(s)

def dense(transposed):
    import torch
    from pyalign_gb300 import autograd as ag
    S = torch.rand(320, 128, 128, device="cuda")
    ag._SOLVERS.clear()
    ag.alignment_score(S.transpose(1, 2) if transposed else S, np.full((320, 2), 128), 0.5, 0.1)
    return launches(next(iter(ag._SOLVERS.values())))

if sys.argv[3] == "letters":
    out = [indexed(4), indexed(5), indexed(5), indexed(4)]
elif sys.argv[3] == "locality":
    out = [aligned("global"), aligned("local")]
else:
    out = [dense(False), dense(True), dense(True), dense(False)]
print("RESULT", json.dumps(out))
"""


def run(kind):
    env = {k: v for k, v in os.environ.items() if not k.startswith("PA_")}
    r = subprocess.run([sys.executable, "-c", RUN, HERE, os.path.dirname(HERE), kind], env=env, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.split("RESULT")[1])


@pytest.mark.parametrize("kind", ["letters", "layout"])
def test_each_kind_is_tuned(kind):
    first, other, again, back = run(kind)
    assert first > 12 and other > 12, (first, other, again, back)
    assert again <= 6 and back <= 6, (first, other, again, back)


def test_local_alignments_are_tried_in_int32():
    """2,100 pairs of 380: global alignments are sure to gain from 16 bits, local ones are timed in
    both (four widths each, twice)."""
    globals_, locals_ = run("locality")
    assert locals_ >= globals_ + 6, (globals_, locals_)
