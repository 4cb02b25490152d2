"""The tiled general-gap sweep (32 x 32 tiles) at the edges of its tiles against the oracle, bit
for bit: lengths around multiples of 32, every locality, direction and input form, gap costs
with many ties, cells of -inf; scores alone and scores with alignments."""

import zlib

import numpy as np
import pytest

from _cases import Gap, call, compare, dense_of, options, pack

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (1, 70), (70, 1), (0, 5), (5, 0), (31, 33), (32, 32), (33, 31), (64, 64), (65, 96), (97, 63),
          (130, 40), (40, 130)]


@pytest.mark.parametrize("locality", ["local", "global", "semiglobal"])
@pytest.mark.parametrize("direction", ["maximize", "minimize"])
@pytest.mark.parametrize("form,gap", [("indexed", Gap("log", 3.0, 1.0)), ("indexed", Gap("log", 1.0, 0.0)),
                                      ("binary", Gap("log", 2.0, 0.5)), ("dense", Gap("log", 1.0, 0.25)),
                                      ("masked", Gap("log", 1.5, 0.5))])
def test_tile_edges(oracle_alg, locality, direction, form, gap):
    from pyalign_gb300 import algorithm as gpu_alg
    rng = np.random.default_rng(zlib.crc32(f"tiles/{locality}/{direction}/{form}/{gap}".encode()))
    pairs = []
    for k, (n, m) in enumerate(SHAPES):
        s = rng.integers(0, 4, n).astype(np.uint32)
        t = np.resize(s, m) if k % 2 and n else rng.integers(0, 4, m).astype(np.uint32)
        flip = rng.random(m) < 0.15
        t = np.where(flip, rng.integers(0, 4, m), t).astype(np.uint32)
        pairs.append((s, t))
    a, b, ln = pack(pairs, len(pairs))
    sign = 1.0 if direction == "maximize" else -1.0
    table = rng.integers(-3, 4, size=(4, 4)).astype(np.float32) * sign
    np.fill_diagonal(table, 3.0 * sign)
    sim = dense_of(a, b, ln, table)
    if form == "dense":
        sim = sim + rng.random(sim.shape).astype(np.float32)
    elif form == "masked":  # cells that may not align
        sim = np.where(rng.random(sim.shape) < 0.3, np.float32(-np.inf * sign), sim).astype(np.float32)
        form = "dense"
    for method, detail in (("score", "score"), ("alignment", "alignment")):
        o = options(gpu_alg, locality=locality, direction=direction, detail=detail, gap=gap, batch_size=len(pairs))
        args = (o, (a.shape[1], b.shape[1]), method, form, a, b, ln, table, sign, -sign, sim)
        _, g = call(gpu_alg, *args)
        _, r = call(oracle_alg, *args)
        assert compare(method, g, r, len(pairs)) is None
