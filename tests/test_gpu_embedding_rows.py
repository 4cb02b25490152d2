"""Embedding alignment with numbers of rows that are no multiple of 4 (needs a GPU): bit for bit the
scores of the similarity the same product gives, through alignment_score -- the border costs of a
global alignment round by the solver's number of rows, so padding S must not change that."""

import numpy as np
import pytest
import torch

from pyalign_gb300 import autograd as ag

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(41, 41), (42, 30), (43, 50), (44, 44), (51, 51), (769, 100)])
@pytest.mark.parametrize("dim", [64, 50])  # the product from float rows, and through stored factors
@pytest.mark.parametrize("locality", ["global", "local", "semiglobal"])
def test_scores_are_those_of_the_similarity(n, m, dim, locality):
    B = 200 if n < 100 else 20
    g = torch.Generator(device="cuda").manual_seed(n)
    Es, Et = torch.randn(B, n, dim, generator=g, device="cuda"), torch.randn(B, m, dim, generator=g, device="cuda")
    rng = np.random.default_rng(n)
    lengths = np.stack([rng.integers(1, n + 1, B), rng.integers(1, m + 1, B)], 1)
    with torch.no_grad():
        got = ag.embedding_alignment_score(Es, Et, lengths, 0.5, 0.1, locality)
        want = ag.alignment_score(ag.cosine_similarity_batch(Es, Et, lengths), lengths, 0.5, 0.1, locality)
    assert torch.equal(got, want)
