"""What alignment scores keep between calls belongs to one thread and one stream: a solver's buffers and
a cached index array may still be in use, or not yet written, by work queued elsewhere."""

import threading

import numpy as np
import pytest

from pyalign_gb300 import autograd as ag

ARGS = (4, 30, 30, "global", "maximize", False, (0.5, 0.1))


def test_solvers_of_streams_and_threads():
    ag._SOLVERS.clear()
    one = ag._solver(*ARGS, 11)
    assert ag._solver(*ARGS, 11) is one
    assert ag._solver(*ARGS, 12) is not one
    other = []
    t = threading.Thread(target=lambda: other.append(ag._solver(*ARGS, 11)))
    t.start()
    t.join()
    assert other[0] is not one
    ag._SOLVERS.clear()


@pytest.mark.gpu
def test_cached_arrays_of_streams():
    import torch
    arr = np.arange(1000, dtype=np.int32)
    a = ag._to_device(arr, "cuda")
    assert ag._to_device(arr, "cuda") is a
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        b = ag._to_device(arr, "cuda")
        assert b is not a and ag._to_device(arr, "cuda") is b
    torch.cuda.synchronize()
    assert torch.equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [False, True])
def test_two_streams_at_once(threads):
    """Two users of one shape, each with its own data and stream, against one after the other."""
    import torch
    n, size, dim, steps = 48, 120, 64, 40
    rng = np.random.default_rng(0)

    def data(user, step):
        g = torch.Generator(device="cuda").manual_seed(100 * user + step)
        r = np.random.default_rng(1000 * user + step)
        return [torch.randn(n, size, dim, generator=g, device="cuda", requires_grad=True) for _ in range(2)], \
            r.integers(1, size + 1, (n, 2)), torch.rand(n, size, size, generator=g, device="cuda")

    def work(x, lengths, S):
        score = ag.embedding_alignment_score(*x, lengths, 0.5, 0.1)
        return [score.detach(), *torch.autograd.grad(score.sum(), x), ag.alignment_score(S, lengths, 0.5, 0.1, "local")]

    inputs = {(u, k): data(u, k) for u in range(2) for k in range(steps)}
    want = {key: work(*v) for key, v in inputs.items()}
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    got, errors = {}, []

    def run(user):
        try:
            with torch.cuda.stream(streams[user]):
                for k in range(steps):
                    got[user, k] = work(*inputs[user, k])
        except BaseException as e:  # noqa: BLE001
            errors.append(repr(e))

    if threads:
        ts = [threading.Thread(target=run, args=(u,)) for u in range(2)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    else:
        for k in rng.permutation(steps):
            for u in range(2):
                with torch.cuda.stream(streams[u]):
                    got[u, k] = work(*inputs[u, k])
    torch.cuda.synchronize()
    assert not errors, errors
    for key, w in want.items():
        for x, y in zip(got[key], w):
            assert torch.equal(x, y), key


@pytest.mark.gpu
def test_the_current_stream_is_the_default():
    import torch
    with torch.cuda.stream(torch.cuda.Stream()):
        assert ag._solver(*ARGS) is ag._solver(*ARGS, torch.cuda.current_stream().cuda_stream)
