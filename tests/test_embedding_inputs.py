"""Embedding alignment refuses factors that do not lie on one CUDA device, or that are not
(batch, len, d), before any pointer reaches a kernel."""

import numpy as np
import pytest
import torch

from pyalign_gb300 import autograd as ag

LENGTHS = np.array([[3, 4]], np.int32)


def refused(Es, Et):
    with pytest.raises(ValueError, match="CUDA tensors on one device"):
        ag.embedding_alignment_score(Es, Et, LENGTHS, 0.5, 0.1)


def test_host_tensors():
    refused(torch.zeros(1, 4, 16), torch.zeros(1, 4, 16))


@pytest.mark.gpu
@pytest.mark.parametrize("dim", [16, 20, 512])  # the product from float rows, and through stored factors
def test_one_host_tensor_or_a_dimension_too_many(dim):
    x = torch.zeros(1, 4, dim, device="cuda")
    refused(x, x.cpu())
    refused(x.cpu(), x)
    refused(x, x[..., None])
    refused(x[..., None], x)
    refused(x[0], x)
    assert ag.embedding_alignment_score(x, x, LENGTHS, 0.5, 0.1).shape == (1,)
