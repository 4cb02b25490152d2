"""A dense similarity copied to the DP's layout (needs a GPU): the same scores and gradients as when it
is read in place, for few long pairs and many short ones; the copy takes room of torch's allocator
for the call alone, and a call that fits without it still fits."""

import numpy as np
import pytest
import torch

from pyalign_gb300 import autograd as ag

pytestmark = pytest.mark.gpu


def run(S, lengths, locality):
    S = S.detach().requires_grad_(True)
    score = ag.alignment_score(S, lengths, 0.5, 0.1, locality)
    return score.detach(), torch.autograd.grad(score.sum(), S)[0]


# pairs, rows, columns: around the 32-column strips and 64-row parts, grids of one part and of many
@pytest.mark.parametrize("B,n,m", [(1, 1, 1), (1, 63, 33), (1, 1203, 1500), (3, 700, 2049), (2, 2050, 65), (40, 129, 257),
                                   (300, 130, 131), (1300, 65, 31)])
@pytest.mark.parametrize("layout", ["along t", "along s, odd pitch", "along t, odd start"])
@pytest.mark.parametrize("locality", ["local", "global"])
def test_copied_and_read_in_place(monkeypatch, B, n, m, layout, locality):
    g = torch.Generator(device="cuda").manual_seed(B + n)
    if layout == "along s, odd pitch":
        S = (torch.rand(B, m, n | 1, generator=g, device="cuda") * 2 - 1).transpose(1, 2)[:, :n]
    elif layout == "along t, odd start":
        S = (torch.rand(B * n * m + 1, generator=g, device="cuda") * 2 - 1)[1:].view(B, n, m)
    else:
        S = torch.rand(B, n, m, generator=g, device="cuda") * 2 - 1
    rng = np.random.default_rng(n)
    lengths = np.stack([rng.integers((n + 1) // 2, n + 1, B), rng.integers((m + 1) // 2, m + 1, B)], 1)
    rooms = []
    room = ag._dense_work
    monkeypatch.setattr(ag, "_dense_work", lambda *a: rooms.append(room(*a)) or rooms[-1])
    got = run(S, lengths, locality)
    assert len(rooms) == 1 and rooms[0] is not None
    monkeypatch.setattr(ag, "_dense_work", lambda *a: None)
    want = run(S, lengths, locality)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def _large():
    ag._SOLVERS.clear()
    torch.cuda.empty_cache()
    S = torch.rand(64, 1000, 1000, device="cuda")  # 256 MB; its traceback words take 40
    return S, np.full((64, 2), 1000), S.numel() * 4


def test_no_copy_is_kept(monkeypatch):
    monkeypatch.setenv("PA_TUNE", "0")
    S, lengths, size = _large()
    free = torch.cuda.mem_get_info()[0]
    with torch.no_grad():
        ag.alignment_score(S, lengths, 0.5, 0.1)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    assert free - torch.cuda.mem_get_info()[0] < size // 2


@pytest.mark.parametrize("share", [1.06, 1.3])
def test_fits_where_it_fits_without_the_copy(monkeypatch, share):
    """Free memory for the copy and little else: room enough to read S in place."""
    monkeypatch.setenv("PA_TUNE", "0")
    S, lengths, size = _large()
    with torch.no_grad():
        want = ag.alignment_score(S, lengths, 0.5, 0.1)
        torch.cuda.synchronize()
        ag._SOLVERS.clear()
        torch.cuda.empty_cache()
        fill = torch.empty(torch.cuda.mem_get_info()[0] - int(share * size), dtype=torch.uint8, device="cuda")
        got = ag.alignment_score(S, lengths, 0.5, 0.1)
        torch.cuda.synchronize()
        del fill
    assert torch.equal(got, want)
    torch.cuda.empty_cache()
