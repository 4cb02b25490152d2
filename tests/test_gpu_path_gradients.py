"""pa_path_gradients on made-up paths at the edges of its 32-step chunks, against a plain
loop over the steps (aligned cells and gap counts are whole numbers: equal, not close)."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make_path(rng, steps, stop):
    """A path of `steps` steps up-left; `stop` ends it at a negative coordinate."""
    pts = [(4 * steps + 3, 4 * steps + 5)]
    for _ in range(steps):
        u, v = pts[-1]
        kind = rng.integers(0, 4)
        d = int(rng.integers(1, 4))
        pts.append((u - 1, v - 1) if kind < 2 else (u - d, v) if kind == 2 else (u, v - d))
    if stop:
        pts.append((-1, pts[-1][1]))
    return np.array(pts, np.int32)


def expected(path, g, shape, dtw, glob):
    dS = np.zeros(shape, np.float32)
    n = [0, 0, 0, 0]
    for (u0, v0), (u1, v1) in zip(path[:-1], path[1:]):
        if u0 < 0 or v0 < 0:
            break
        if dtw or (u1 == u0 - 1 and v1 == v0 - 1):
            dS[u0, v0] += g
        elif v1 == v0 and u1 < u0:
            n[0] += 1
            n[1] += u0 - u1 - 1
        elif u1 == u0 and v1 < v0:
            n[2] += 1
            n[3] += v0 - v1 - 1
    if len(path) and glob and not dtw:
        u, v = path[-1]
        if u < 0 <= v:
            n[2] += 1
            n[3] += v
        elif v < 0 <= u:
            n[0] += 1
            n[1] += u
    return dS, np.float32(-g) * np.array(n, np.float32)


@pytest.mark.parametrize("dtw", [False, True])
@pytest.mark.parametrize("stop", [False, True])
def test_chunk_edges(dtw, stop):
    import torch
    from pyalign_gb300 import algorithm as alg
    from pyalign_gb300 import autograd as ag
    rng = np.random.default_rng(5)
    sizes = [0, 1, 2, 30, 31, 32, 33, 62, 63, 64, 65, 97, 130]
    paths = [make_path(rng, s, stop) for s in sizes] + [np.zeros((0, 2), np.int32)]
    B = len(paths)
    n = 4 * max(sizes) + 8
    off = np.zeros(B, np.int64)
    off[1:] = np.cumsum([2 * len(p) for p in paths])[:-1]
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    flat, offd = dev(np.concatenate([p.ravel() for p in paths])), dev(off)
    plen = dev(np.array([len(p) for p in paths], np.int32))
    grad = rng.random(B).astype(np.float32)
    gd = dev(grad)
    dS = torch.zeros(B, n, n, device="cuda")
    so = dev(np.arange(B, dtype=np.int64) * n * n)
    dgap = torch.full((B, 4), 7.0, device="cuda")
    alg.check(ag._lib().pa_path_gradients(
        1 if dtw else 0, 1, 1, B, flat.data_ptr(), offd.data_ptr(), plen.data_ptr(), gd.data_ptr(), dS.data_ptr(),
        so.data_ptr(), n, 1, dgap.data_ptr(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    for k, p in enumerate(paths):
        e_s, e_g = expected(p, grad[k], (n, n), dtw, True)
        assert np.array_equal(dS[k].cpu().numpy(), e_s), sizes[min(k, len(sizes) - 1)]
        assert np.array_equal(dgap[k].cpu().numpy(), e_g), sizes[min(k, len(sizes) - 1)]
