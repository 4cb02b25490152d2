"""The similarity product from float rows and the path gradients that go with it (need a GPU).

pa_similarity_rows normalises float rows on the way into the tensor cores: the BF16 factors are
those of pa_normalize_rows_bf16 bit for bit, so 1 / |E| is equal and the product matches
pa_similarity_bf16 up to the order of float32 additions (unit rows: 2^-24 per term, dim terms).
Only cells inside the lengths may be written.  pa_path_embedding_gradients_rows rounds the
factors again from the rows: it must match pa_path_embedding_gradients_full up to the order in
which the dim terms of g . en are added, and write every row.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [[300, 520], [1, 1], [127, 256], [128, 257], [129, 255], [0, 50], [50, 0], [257, 3], [5, 513], [300, 128],
           [16, 129]]


@pytest.fixture(scope="module")
def torch_ag():
    torch = pytest.importorskip("torch")
    from pyalign_gb300 import build
    build.build()
    if not torch.cuda.is_available():
        pytest.fail("no CUDA device visible")
    from pyalign_gb300 import autograd
    return torch, autograd


def _rows(torch, dim, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    B = len(LENGTHS)
    Es = torch.randn(B, 300, dim, device="cuda", generator=g)
    Et = torch.randn(B, 520, dim, device="cuda", generator=g)
    Es[0, 3] = 0.0       # a zero row: 1 / |E| is capped
    Es[4, 129:] = float("nan")  # past the length: not read
    return Es, Et


@pytest.mark.parametrize("normalize", [True, False])
@pytest.mark.parametrize("dim", [4, 16, 20, 64, 100, 128, 132, 192, 256])
def test_product_and_norms_match_the_stored_factors(torch_ag, dim, normalize):
    torch, ag = torch_ag
    Es, Et = _rows(torch, dim, dim)
    lengths = np.array(LENGTHS)
    B, n_s, n_t = len(lengths), Es.shape[1], Et.shape[1]
    out = torch.full((B, n_t, n_s), float("nan"), device="cuda")
    inv_s, inv_t = ag._similarity_rows(Es, Et, lengths, normalize, out)
    Esb, ws = ag.normalized_bf16(Es, normalize, lengths[:, 0])
    Etb, wt = ag.normalized_bf16(Et, normalize, lengths[:, 1])
    want = ag.similarity_bf16(Esb, Etb, lengths, out=torch.full((B, n_t, n_s), float("nan"), device="cuda"))
    assert ag.tensor_core_status() == 0
    got = out.transpose(1, 2)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    for k, (ls, lt) in enumerate(lengths):
        if ls == 0 or lt == 0:
            continue
        assert torch.equal(inv_s.view(B, n_s)[k, :ls], ws.view(B, n_s)[k, :ls])
        assert torch.equal(inv_t.view(B, n_t)[k, :lt], wt.view(B, n_t)[k, :lt])
        bound = torch.outer(Esb[k, :ls].float().norm(dim=1), Etb[k, :lt].float().norm(dim=1)) * dim * 2.0 ** -23
        assert ((got[k, :ls, :lt] - want[k, :ls, :lt]).abs() <= bound).all(), k


def test_many_pairs_walk_over_several_ranges(torch_ag):
    """More tiles than CTAs, empty pairs between, ranges that begin inside a pair."""
    torch, ag = torch_ag
    rng = np.random.default_rng(3)
    B, n, dim = 700, 400, 64
    lengths = rng.integers(0, n + 1, size=(B, 2)) * (rng.random((B, 1)) < 0.8)
    g = torch.Generator(device="cuda").manual_seed(3)
    Es, Et = (torch.randn(B, n, dim, device="cuda", generator=g) for _ in range(2))
    out = torch.full((B, n, n), float("nan"), device="cuda")
    ag._similarity_rows(Es, Et, lengths, True, out)
    want = torch.bmm(torch.nn.functional.normalize(Et, dim=2), torch.nn.functional.normalize(Es, dim=2).transpose(1, 2))
    inside = (torch.arange(n, device="cuda")[None, :, None] < torch.tensor(lengths[:, 1], device="cuda")[:, None, None]) \
        & (torch.arange(n, device="cuda")[None, None, :] < torch.tensor(lengths[:, 0], device="cuda")[:, None, None])
    assert ag.tensor_core_status() == 0
    assert torch.equal(torch.isnan(out), ~inside)
    # two factors rounded to BF16 (2^-9 each) of unit rows
    assert (out[inside] - want[inside]).abs().max() <= 2.0 ** -7


@pytest.mark.parametrize("normalize", [True, False])
@pytest.mark.parametrize("dim", [4, 20, 100, 128, 132, 256])
def test_gradients_match_the_stored_factors(torch_ag, dim, normalize):
    torch, ag = torch_ag
    Es, Et = _rows(torch, dim, 1000 + dim)
    lengths = np.array(LENGTHS)
    B, n_s, n_t = len(lengths), Es.shape[1], Et.shape[1]
    St = torch.zeros((B, n_t, n_s), device="cuda")
    inv_s, inv_t = ag._similarity_rows(Es, Et, lengths, normalize, St)
    scores, paths, plen, poff, _ = ag._forward_paths(St.transpose(1, 2), lengths, (0.5, 0.1), "global", "maximize", False)
    grad = torch.rand(B, device="cuda") + 0.5
    stream = torch.cuda.current_stream().cuda_stream
    walk = (paths.data_ptr(), poff.data_ptr(), plen.data_ptr(), grad.data_ptr())
    got = [torch.full_like(x, float("nan")) for x in (Es, Et)]
    ag._alg.check(ag._lib().pa_path_embedding_gradients_rows(
        B, dim, int(normalize), *walk, Es.data_ptr(), Et.data_ptr(), inv_s.data_ptr(), inv_t.data_ptr(), n_s, n_t,
        got[0].data_ptr(), got[1].data_ptr(), stream))
    Ps, Pt = ag._pad16(Es), ag._pad16(Et)
    Esb, ws = ag.normalized_bf16(Ps, normalize, lengths[:, 0])
    Etb, wt = ag.normalized_bf16(Pt, normalize, lengths[:, 1])
    want = [torch.full_like(x, float("nan")) for x in (Ps, Pt)]
    ag._alg.check(ag._lib().pa_path_embedding_gradients_full(
        B, Ps.shape[2], int(normalize), *walk, Ps.data_ptr(), Pt.data_ptr(), Esb.data_ptr(), Etb.data_ptr(),
        ws.data_ptr(), wt.data_ptr(), n_s, n_t, want[0].data_ptr(), want[1].data_ptr(), stream))
    for a, b, w, n in ((got[0], want[0], ws, n_s), (got[1], want[1], wt, n_t)):
        b = b[..., :dim]
        assert not torch.isnan(a).any()
        assert torch.equal(a == 0, b == 0) or normalize
        # g . en differs by at most dim roundings of g (unit rows), times |en| <= 1 and 1 / |E|
        bound = (grad.view(B, 1) * w.view(B, n).nan_to_num()).unsqueeze(2) * (dim + 8) * 2.0 ** -23
        assert ((a - b).abs() <= (bound if normalize else torch.zeros_like(bound))).all()
