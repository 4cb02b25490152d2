"""Workloads of the alignment framework for timing and comparison.

A case is one call (or one forward + backward) as a user's program makes it, through the
module's solver methods, pa_solve_batch, or the autograd functions.  `listed()` gives the
standing workloads, `draw(rng)` one more of the same ranges, `prepare` what a program has in
hand before the call, `run` one pass, `work` the bytes and operations the pass cannot do
without, and `exact` the results in 64 bits from plain torch.
"""

import ctypes
import math
import types

import numpy as np
import torch

from pyalign_gb300 import algorithm as alg
from pyalign_gb300 import autograd as ag

P = ctypes.POINTER
NEG = -1e30


# --------------------------------------------------------------------------- cases

def listed():
    return [
        # the module's own call on a handful of short word pairs with a fractional gap cost
        # (float32 scoring), host arrays: an interactive use, latency only
        bag("few_words", kind="module", pairs=8, s=(8, 40), t=(8, 40), letters=20, gap="linear", open=0.5,
            locality="global", codomain="alignment"),
        # 4096 pairs of 64 x 64 letters, equal / unequal scoring, global linear gaps, host
        # arrays in, scores and alignments out: a batch of words, the smallest bag
        bag("words_64", kind="host", pairs=4096, s=(64, 64), t=(64, 64), letters=20, form="binary", gap="linear",
            open=1.0, locality="global", codomain="alignment"),
        # the headline bag: 65,536 DNA pairs of uneven length, half of them mutated copies,
        # local Gotoh, score + alignment, codes on the device
        bag("dna_local", pairs=65536, s=(100, 1000), t=(100, 1000), letters=4, gap="affine", open=5.0, extend=2.0,
            locality="local", codomain="alignment"),
        # reads scored against windows: DNA, local Gotoh, scores only (a filter pass)
        bag("dna_scores", pairs=32768, s=(100, 250), t=(200, 500), letters=4, gap="affine", open=5.0, extend=2.0,
            locality="local", codomain="score"),
        # proteins of ordinary length, 20-letter matrix, global Gotoh, score + alignment
        bag("protein_global", pairs=4096, s=(50, 600), t=(50, 600), letters=20, gap="affine", open=11.0, extend=1.0,
            locality="global", codomain="alignment"),
        # few long pairs, 20-letter matrix, semiglobal Gotoh, scores only
        bag("protein_long", pairs=256, s=(5000, 5000), t=(10000, 10000), letters=20, gap="affine", open=10.0,
            extend=1.0, locality="semiglobal", codomain="score"),
        # every optimal alignment: masks of all pairs, co-optimal path counts, and the first
        # alignments of each pair from its iterator
        bag("all_optimal", kind="all", pairs=16, s=(2000, 3000), t=(3000, 5000), letters=20, gap="affine", open=10.0,
            extend=1.0, locality="semiglobal", codomain="alignment"),
        # a general (logarithmic) gap cost: DNA, local, score + alignment, host arrays
        bag("log_gap", kind="host", pairs=64, s=(300, 300), t=(300, 300), letters=4, gap="log", open=3.0, extend=1.0,
            locality="local", codomain="alignment"),
        # a training step through a dense similarity: scores, dS and the gap gradients
        {"name": "dense_step", "kind": "dense", "pairs": 1024, "lo": 100, "hi": 400, "locality": "local",
         "open": 0.5, "extend": 0.1},
        # a training step on per-token embeddings: cosine on the tensor cores, global Gotoh,
        # gradients of both embeddings and of the gap costs
        {"name": "embed_step", "kind": "embed", "pairs": 4096, "lo": 64, "hi": 256, "dim": 128, "grad": True,
         "open": 0.5, "extend": 0.1},
        # scoring of longer embedding pairs without gradients
        {"name": "embed_scores", "kind": "embed", "pairs": 8192, "lo": 32, "hi": 512, "dim": 256, "grad": False,
         "open": 0.5, "extend": 0.1},
        # a training step of DTW on one-dimensional series
        {"name": "dtw_step", "kind": "series", "pairs": 4096, "lo": 128, "hi": 1024},
    ]


def bag(name, kind="device", pairs=1, s=(1, 1), t=(1, 1), letters=4, form="indexed", gap="linear", open=1.0,
        extend=0.0, locality="global", codomain="score"):
    return {"name": name, "kind": kind, "pairs": pairs, "s_lo": s[0], "s_hi": s[1], "t_lo": t[0], "t_hi": t[1],
            "letters": letters, "form": form, "gap": gap, "open": open, "extend": extend, "locality": locality,
            "codomain": codomain}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a kind, then its sizes, log-uniform where the range is wide."""
    kind = rng.choice(["module", "host", "device", "device", "device", "long", "all", "log", "dense", "embed", "embed",
                       "series"])
    gap = rng.choice(["linear", "affine"])
    open_, ext = (float(rng.randint(1, 4)), 0.0) if gap == "linear" else (float(rng.randint(3, 12)),
                                                                         float(rng.randint(1, 3)))
    locality = rng.choice(["local", "global", "semiglobal"])
    codomain = rng.choice(["score", "alignment"])
    if kind == "module":
        n = _log(rng, 5, 60)
        c = bag("", kind=kind, pairs=rng.randint(1, 16), s=(max(1, n // 2), n), t=(max(1, n // 3), n), letters=20,
                gap=gap, open=open_ - 0.5, extend=max(0.0, ext - 0.75) if gap == "affine" else 0.0,
                locality=locality, codomain="alignment")
    elif kind == "host":
        n, m = _log(rng, 20, 200), _log(rng, 20, 200)
        c = bag("", kind=kind, pairs=_log(rng, 256, 8192), s=(max(1, n // 2), n), t=(max(1, m // 2), m),
                letters=rng.choice([4, 20]), form=rng.choice(["binary", "indexed"]), gap=gap, open=open_, extend=ext,
                locality=locality, codomain=codomain)
    elif kind == "device":
        n, m = _log(rng, 60, 1000), _log(rng, 60, 1000)
        pairs = max(64, min(_log(rng, 1024, 65536), int(1.6e10 / (n * m))))
        c = bag("", pairs=pairs, s=(max(1, n // rng.randint(1, 10)), n), t=(max(1, m // rng.randint(1, 10)), m),
                letters=rng.choice([4, 20]), gap=gap, open=open_, extend=ext, locality=locality, codomain=codomain)
    elif kind == "long":
        n, m = _log(rng, 1500, 6000), _log(rng, 1500, 12000)
        pairs = max(8, min(_log(rng, 16, 256), int(1.2e10 / (n * m))))
        c = bag("", pairs=pairs, s=(n - n // 5, n), t=(m - m // 5, m), letters=rng.choice([4, 20]), gap=gap,
                open=open_, extend=ext, locality=locality, codomain="score")
    elif kind == "all":
        n, m = _log(rng, 300, 3000), _log(rng, 300, 5000)
        c = bag("", kind=kind, pairs=max(4, min(_log(rng, 4, 32), int(2.4e8 / (n * m)))), s=(n // 2 + 1, n),
                t=(m // 2 + 1, m), letters=20, gap="affine", open=10.0, extend=1.0,
                locality=rng.choice(["global", "semiglobal"]), codomain="alignment")
    elif kind == "log":
        n, m = _log(rng, 50, 600), _log(rng, 50, 600)
        pairs = max(2, min(_log(rng, 8, 512), int(3.4e9 / (n * m * (n + m)))))
        c = bag("", kind="host", pairs=pairs, s=(n // 2 + 1, n), t=(m // 2 + 1, m), letters=rng.choice([4, 20]),
                gap="log", open=float(rng.randint(1, 4)), extend=rng.choice([0.5, 1.0, 2.0]), locality=locality,
                codomain=codomain)
    elif kind == "dense":
        n = _log(rng, 40, 500)
        c = {"kind": kind, "pairs": max(32, min(_log(rng, 64, 4096), int(2.0e8 / (n * n)))), "lo": max(1, n // 4),
             "hi": n, "locality": locality, "open": rng.choice([0.5, 0.8]), "extend": rng.choice([0.1, 0.25])}
    elif kind == "embed":
        n, dim = _log(rng, 40, 512), rng.choice([64, 100, 128, 256])
        grad = rng.random() < 0.6
        pairs = max(64, min(_log(rng, 256, 8192), int((1.3e8 if grad else 1.0e9) / (n * dim))))
        c = {"kind": kind, "pairs": pairs, "lo": max(1, n // 4), "hi": n, "dim": dim, "grad": grad, "open": 0.5,
             "extend": 0.1}
    else:
        n = _log(rng, 64, 1024)
        c = {"kind": kind, "pairs": max(64, min(_log(rng, 256, 8192), int(4.2e9 / (n * n)))), "lo": max(1, n // 8),
             "hi": n}
    c.pop("name", None)
    return c


# --------------------------------------------------------------------------- inputs

class _Linear:
    def __init__(self, g):
        self.g = g

    def to_special_case(self):
        return {"linear": self.g}


class _Affine:
    """w(k) = open + extend (k - 1)"""

    def __init__(self, open_, extend):
        self.u, self.v = open_ - extend, extend

    def to_special_case(self):
        return {"affine": (self.u, self.v)}


class _Log:
    """w(k) = u + v ln k"""

    def __init__(self, u, v):
        self.u, self.v = u, v

    def to_special_case(self):
        return {}

    def costs(self, n):
        w = np.full((n,), self.u, dtype=np.float32)
        w[1:] += self.v * np.log(np.arange(1, n), dtype=np.float32)
        w[0] = 0
        return w


def _gap(case):
    if case["gap"] == "linear":
        return _Linear(case["open"])
    if case["gap"] == "affine":
        return _Affine(case["open"], case["extend"])
    return _Log(case["open"], case["extend"])


def _table(case, seed):
    """Letters' similarities: DNA +2 / -3, or a random symmetric integer matrix (diagonal
    4..11, off-diagonal -4..2); the binary form's +1 / -1 as a table."""
    k = case["letters"]
    if case["form"] == "binary":
        return np.where(np.eye(k, dtype=bool), 1.0, -1.0).astype(np.float32)
    if k == 4:
        return np.where(np.eye(4, dtype=bool), 2.0, -3.0).astype(np.float32)
    r = np.random.RandomState(seed % (1 << 31) + 17)
    m = r.randint(-4, 3, (k, k))
    m = np.triu(m, 1) + np.triu(m, 1).T
    np.fill_diagonal(m, r.randint(4, 12, k))
    return m.astype(np.float32)


def _codes(case, seed):
    """Code rows (pairs, n) int32 on the device and host lengths (2, pairs): odd pairs are a
    sequence and a copy of it with about 10% substitutions and indels, cut to t's range."""
    B, ns, nt, k = case["pairs"], case["s_hi"], case["t_hi"], case["letters"]
    r = np.random.RandomState(seed % (1 << 31))
    ls = r.randint(case["s_lo"], ns + 1, B).astype(np.int32)
    lt = r.randint(case["t_lo"], nt + 1, B).astype(np.int32)
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randint(0, k, (B, ns), generator=g, device="cuda", dtype=torch.int32)
    b = torch.randint(0, k, (B, nt), generator=g, device="cuda", dtype=torch.int32)
    x = torch.rand(B, nt, generator=g, device="cuda")
    step = (x < 0.025).int() - ((x > 0.025) & (x < 0.05)).int()
    src = torch.arange(nt, device="cuda") + torch.cumsum(step, 1)
    copied = torch.gather(a, 1, src.clamp(0, ns - 1))
    related = ((torch.arange(B, device="cuda") % 2 == 1)[:, None]) & (x < 0.95) & (src >= 0) & (src < ns)
    b = torch.where(related, copied, b)
    lt[1::2] = np.clip(ls[1::2], case["t_lo"], nt)
    return a, b, np.ascontiguousarray(np.stack([ls, lt]))


def _solver(case, n_s, n_t):
    mod = alg.m16 if max(n_s, n_t) < 16000 else alg.m32
    every = case["kind"] == "all"
    return mod.create_solver(n_s, n_t, mod.create_options({
        "solver": alg.Type.ALIGNMENT, "direction": alg.Direction.MAXIMIZE, "batch": True,
        "batch_size": case["pairs"], "return_dup": False,
        "locality": alg.Locality.__members__[case["locality"].upper()],
        "codomain": types.SimpleNamespace(detail=alg.Detail.__members__[case["codomain"].upper()],
                                          count=alg.Count.ALL if every else alg.Count.ONE),
        "gap_cost": _gap(case)}))


def _lengths(case, seed):
    r = np.random.RandomState(seed % (1 << 31))
    return r.randint(case["lo"], case["hi"] + 1, (case["pairs"], 2))


def _floats(case, seed):
    """The tensors of the differentiable kinds."""
    B, n = case["pairs"], case["hi"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "dense":
        return (torch.rand(B, n, n, generator=g, device="cuda") * 2 - 1,)
    if case["kind"] == "embed":
        return tuple(torch.randn(B, n, case["dim"], generator=g, device="cuda") for _ in range(2))
    return tuple(torch.cumsum(torch.randn(B, n, generator=g, device="cuda"), 1) for _ in range(2))


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("dense", "embed", "series"):
        state = {"case": case, "lengths": _lengths(case, seed),
                 "x": [v.requires_grad_(bool(case.get("grad", True))) for v in _floats(case, seed)]}
        if kind != "series" and case.get("grad", True):
            # learned gap costs
            state["gap"] = [torch.tensor(case[k], requires_grad=True) for k in ("open", "extend")]
            state["x"] += state["gap"]
        if case.get("grad", True):
            g = torch.Generator(device="cuda").manual_seed(seed + 1)
            state["up"] = torch.rand(case["pairs"], generator=g, device="cuda") + 0.5
        return state
    a, b, length = _codes(case, seed)
    B, n_s, n_t = case["pairs"], case["s_hi"], case["t_hi"]
    table = _table(case, seed)
    solver = _solver(case, n_s, n_t)
    state = {"case": case, "solver": solver, "table": table, "length": length}
    if kind in ("module", "all"):
        state["a"], state["b"] = a.cpu().numpy().astype(np.uint32), b.cpu().numpy().astype(np.uint32)
        state["length"] = length.astype(np.uint16)
        return state
    sizes = np.minimum(length[0], length[1]).astype(np.int64)
    offs = np.zeros(B, np.int64)
    offs[1:] = np.cumsum(sizes)[:-1]
    room = B * min(n_s, n_t)  # the maps lie packed at its start
    dev = kind == "device"
    if dev:
        tab = torch.from_numpy(table).cuda()
        scores = torch.empty(B, dtype=torch.float32, device="cuda")
        maps = torch.full((room,), -1, dtype=torch.int32, device="cuda")
        ptr = lambda x: x.data_ptr()  # noqa: E731
        alg.check(alg.lib().pa_solver_set_stream(solver.handle,
                                                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    else:
        a, b = a.cpu().numpy().astype(np.uint32), b.cpu().numpy().astype(np.uint32)
        tab, scores = table, np.empty(B, np.float32)
        maps = np.full(room, -1, np.int32)
        ptr = lambda x: x.ctypes.data  # noqa: E731
    if case["codomain"] == "score":
        maps = None
    binary = case["form"] == "binary"
    batch = alg.Batch(form=2 if binary else 1, location=1 if dev else 0, batch=B, n_s=n_s, n_t=n_t,
                      a=ctypes.cast(ptr(a), P(ctypes.c_uint32)), b=ctypes.cast(ptr(b), P(ctypes.c_uint32)),
                      table=None if binary else ctypes.cast(ptr(tab), P(ctypes.c_float)),
                      table_rows=0 if binary else table.shape[0], table_cols=0 if binary else table.shape[1],
                      eq=1.0 if binary else 0.0, ne=-1.0 if binary else 0.0,
                      length=length.ctypes.data_as(P(ctypes.c_int32)))
    state.update(a=a, b=b, tab=tab, scores=scores, maps=maps, offs=offs, batch=batch, scores_p=ptr(scores),
                 maps_p=None if maps is None else ptr(maps), offs_p=offs.ctypes.data_as(P(ctypes.c_int64)))
    return state


# --------------------------------------------------------------------------- one pass

FIRST = 5  # alignments a program takes from each lane's iterator


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("dense", "embed", "series"):
        x = state["x"]
        gap = state.get("gap", (case.get("open"), case.get("extend")))
        with torch.set_grad_enabled("up" in state):
            if kind == "dense":
                score = ag.alignment_score(x[0], state["lengths"], gap[0], gap[1], case["locality"], "maximize")
            elif kind == "embed":
                score = ag.embedding_alignment_score(x[0], x[1], state["lengths"], gap[0], gap[1])
            else:
                score = ag.dtw_series_score(x[0], x[1], state["lengths"])
        if "up" not in state:
            return {"scores": score}
        grads = torch.autograd.grad(score, x, state["up"])
        return {"scores": score.detach(), "grads": list(grads)}
    if kind == "module":
        lanes = state["solver"].solve_indexed_for_alignment(state["a"], state["b"], state["table"], state["length"])
        maps = np.full((len(lanes), case["s_hi"]), -1, np.int16)
        for row, x in zip(maps, lanes):
            row[:len(x.s_to_t)] = x.s_to_t
        return {"scores": np.array([x.score for x in lanes], np.float32), "s_to_t": maps}
    if kind == "all":
        lanes = state["solver"].solve_indexed_for_alignment_iterator(state["a"], state["b"], state["table"],
                                                                     state["length"])
        counts = np.array([it.path_count() for it in lanes], np.uint64)
        scores = np.zeros((len(lanes), FIRST), np.float32)
        maps = np.full((len(lanes), FIRST, case["s_hi"]), -1, np.int16)
        for lane, it in enumerate(lanes):
            for k in range(FIRST):
                x = it.next()
                if x is None:
                    break
                scores[lane, k] = x.score
                maps[lane, k, :len(x.s_to_t)] = x.s_to_t
        return {"counts": counts, "scores": scores, "s_to_t": maps}
    alg.check(alg.lib().pa_solve_batch(state["solver"].handle, ctypes.byref(state["batch"]), state["scores_p"],
                                       state["maps_p"], state["offs_p"]))
    return {"scores": state["scores"]} if state["maps"] is None else {"scores": state["scores"],
                                                                       "maps": state["maps"]}


def work(case):
    """Bytes of the inputs and outputs once each, and the recurrence's operations."""
    B = case["pairs"]
    if case["kind"] in ("dense", "embed", "series"):
        lo, hi = case["lo"], case["hi"]
        n = (lo + hi) / 2
        cells = B * n * n
        grad = case.get("grad", True)
        if case["kind"] == "dense":  # S inside the lengths, dS whole
            return {"bytes": 4 * cells + 4 * B * hi * hi, "flops": 13 * cells}
        if case["kind"] == "embed":
            d = case["dim"]
            rows = 2 * B * n * d * 4
            return {"bytes": rows + (2 * B * hi * d * 4 if grad else 0), "flops": (2 * d + 13) * cells}
        return {"bytes": 2 * B * n * 4 + 2 * B * hi * 4, "flops": 5 * cells}
    ms, mt = (case["s_lo"] + case["s_hi"]) / 2, (case["t_lo"] + case["t_hi"]) / 2
    aligned = case["codomain"] == "alignment"
    cells = B * ms * mt
    nbytes = B * 4 * (ms + mt) + B * 4 + (B * 4 * min(ms, mt) if aligned else 0)
    if case["kind"] == "all":  # the map of each alignment taken, and a count, per pair
        return {"bytes": nbytes + FIRST * B * 4 * ms + 8 * B, "flops": 17 * cells}
    per = {"linear": 5, "affine": 9}.get(case["gap"], ms + mt + 2)
    per = per + (case["locality"] == "local") + (4 if aligned and case["gap"] != "log" else 0)
    return {"bytes": nbytes, "flops": per * cells}


# --------------------------------------------------------------------------- 64 bits

def _wavefront(diag, ls, lt, gap, locality, codes=False):
    """Optimal scores in 64 bits over anti-diagonals (maximising): diag(d, i0, i1) gives
    S(i, d - i) for i0 <= i < i1 of every pair; gap is ("linear", g), ("affine", open,
    extend) or None for DTW.  With `codes`, also every cell's traceback code per diagonal
    (bits 0-1: 3 stop, 2 diagonal, 1 up, 0 left; bit 2 / 3: the vertical / horizontal gap
    extends) and the seed cells."""
    dev = ls.device
    B, ns, nt = ls.numel(), int(ls.max()), int(lt.max())
    f = lambda *s: torch.full(s, NEG, dtype=torch.float64, device=dev)  # noqa: E731
    if gap is None:
        w = lambda k: 0.0 if k == 0 else -NEG  # noqa: E731
        op = ex = 0.0
    elif gap[0] == "linear":
        w = lambda k: gap[1] * k if locality == "global" else 0.0  # noqa: E731
        op = ex = gap[1]
    else:
        op, ex = gap[1], gap[2]
        w = lambda k: (op + ex * (k - 1) if k else 0.0) if locality == "global" else 0.0  # noqa: E731
    # D of diagonals d - 1 and d - 2, index i + 1 for row i (row -1 and column -1 are borders)
    D1, D2, Pv, Qh = f(B, ns + 1), f(B, ns + 1), f(B, ns + 1), f(B, ns + 1)
    D2[:, 0] = 0.0
    D1[:, 0] = D1[:, 1] = -w(1)
    best, bi, bj = f(B), torch.zeros_like(ls), torch.zeros_like(ls)
    all_codes = []
    rows = torch.arange(ns, device=dev)
    last = (ls + lt - 2).long()
    for d in range(ns + nt - 1):
        i0, i1 = max(0, d - nt + 1), min(ns, d + 1)
        S = diag(d, i0, i1)
        up, left, dg = D1[:, i0:i1], D1[:, i0 + 1:i1 + 1], D2[:, i0:i1]
        if gap is None:
            pe = qe = None
            p, q = up, left
            dd = dg
        elif gap[0] == "linear":
            pe = qe = None
            p, q, dd = up - op, left - op, dg + S
        else:
            oP, eP, oQ, eQ = up - op, Pv[:, i0:i1] - ex, left - op, Qh[:, i0 + 1:i1 + 1] - ex
            p, q, dd = torch.maximum(oP, eP), torch.maximum(oQ, eQ), dg + S
            pe, qe = eP > oP, eQ > oQ
        v = torch.maximum(torch.maximum(p, q), dd)
        if locality == "local":
            v = v.clamp_min(0.0)
        if codes:
            c = torch.where(dd >= torch.maximum(p, q), 2, torch.where(p >= q, 1, 0))
            if locality == "local":
                c = torch.where(v <= 0.0, 3, c)
            if pe is not None:
                c = c + 4 * pe + 8 * qe
            all_codes.append((i0, c.to(torch.int8)))
        if gap is None:
            v = v + S
        D = f(B, ns + 1)
        D[:, i0 + 1:i1 + 1] = v
        if d + 1 < nt:
            D[:, 0] = -w(d + 2)
        if d + 1 < ns:
            D[:, d + 2] = -w(d + 2)
        if gap is not None and gap[0] == "affine":
            Pn, Qn = f(B, ns + 1), f(B, ns + 1)
            Pn[:, i0 + 1:i1 + 1], Qn[:, i0 + 1:i1 + 1] = p, q
            Pv, Qh = Pn, Qn
        r = rows[i0:i1]
        if locality == "global":
            hit = torch.where(last == d, v.gather(1, (ls - 1 - i0).clamp(0, i1 - i0 - 1).long()[:, None])[:, 0], best)
            best = hit
        else:
            ok = (r[None] < ls[:, None]) & (d - r[None] < lt[:, None])
            if locality == "semiglobal":
                ok &= (r[None] == ls[:, None] - 1) | (d - r[None] == lt[:, None] - 1)
            m, at = v.masked_fill(~ok, NEG).max(1)
            bi = torch.where(m > best, at + i0, bi)
            bj = torch.where(m > best, d - at - i0, bj)
            best = torch.maximum(best, m)
        D2, D1 = D1, D
    if locality == "global":
        bi, bj = ls - 1, lt - 1
    return (best, all_codes, bi, bj) if codes else best


def _walk(codes, bi, bj, ns, nt, dtw):
    """Follow the codes from the seeds: the visited diagonal cells (all cells for DTW) as
    (pair, i, j) and per pair the opened and extended gap steps."""
    dev = bi.device
    B = bi.numel()
    table = torch.zeros(len(codes), B, ns, dtype=torch.int8, device=dev)
    for d, (i0, c) in enumerate(codes):
        table[d, :, i0:i0 + c.shape[1]] = c
    i, j = bi.long().clone(), bj.long().clone()
    lane = torch.arange(B, device=dev)
    layer = torch.zeros(B, dtype=torch.long, device=dev)  # 0 D, 1 in a vertical gap, 2 horizontal
    live = torch.ones(B, dtype=torch.bool, device=dev)
    cells = []
    opens, exts = torch.zeros(B, dtype=torch.float64, device=dev), torch.zeros(B, dtype=torch.float64, device=dev)
    while True:
        live = live & (i >= 0) & (j >= 0)
        if not bool(live.any()):
            break
        c = table[(i + j).clamp(0, len(codes) - 1), lane, i.clamp_min(0)].long()
        src = c & 3
        live = live & ~((layer == 0) & (src == 3))
        step = torch.where(layer == 0, src, torch.where(layer == 1, 1, 0))  # 2 diagonal, 1 up, 0 left
        mark = live if dtw else live & (step == 2)
        cells.append(torch.stack([lane[mark], i[mark], j[mark]]))
        vertical, horizontal = live & (step == 1), live & (step == 0)
        pe, qe = (c & 4) != 0, (c & 8) != 0
        grow = (vertical & pe) | (horizontal & qe)
        exts += grow.double()
        opens += ((vertical | horizontal) & ~grow).double()
        layer = torch.where(vertical & pe, 1, torch.where(horizontal & qe, 2, 0))
        i = torch.where(live & (step >= 1), i - 1, i)
        j = torch.where(live & (step != 1), j - 1, j)
    return torch.cat(cells, 1), opens, exts, i, j


def _general(S, ls, lt, w, locality):
    """General gap costs in 64 bits: S (B, ns, nt), w the costs of gaps of 0.. letters."""
    B, ns, nt = S.shape
    D = torch.full((B, ns + 1, nt + 1), NEG, dtype=torch.float64, device=S.device)
    border = -w if locality == "global" else torch.zeros_like(w)
    D[:, :, 0], D[:, 0, :] = border[:ns + 1], border[:nt + 1]
    ks, kt = torch.arange(ns + 1, device=S.device), torch.arange(nt + 1, device=S.device)
    for d in range(ns + nt - 1):
        i = torch.arange(max(0, d - nt + 1), min(ns, d + 1), device=S.device)
        j = d - i
        gs, gt = (i + 1)[:, None] - ks, (j + 1)[:, None] - kt
        ws = torch.where(gs > 0, w[gs.clamp_min(0)], -NEG)
        wt = torch.where(gt > 0, w[gt.clamp_min(0)], -NEG)
        v = torch.maximum((D[:, :, j + 1].transpose(1, 2) - ws).amax(2), (D[:, i + 1, :] - wt).amax(2))
        v = torch.maximum(v, D[:, i, j] + S[:, i, j])
        D[:, i + 1, j + 1] = v.clamp_min(0.0) if locality == "local" else v
    D = D[:, 1:, 1:]
    i, j = torch.arange(ns, device=S.device)[None, :, None], torch.arange(nt, device=S.device)[None, None]
    last_i, last_j = i == (ls - 1)[:, None, None], j == (lt - 1)[:, None, None]
    ok = (i < ls[:, None, None]) & (j < lt[:, None, None])
    if locality == "global":
        ok = ok & last_i & last_j
    elif locality == "semiglobal":
        ok = ok & (last_i | last_j)
    return D.masked_fill(~ok, NEG).amax((1, 2))


def exact(case, seed):
    kind = case["kind"]
    if kind == "all":
        return None  # whole numbers and maps
    if kind in ("dense", "embed", "series"):
        return _exact_floats(case, seed)
    a, b, length = _codes(case, seed)
    table = torch.from_numpy(_table(case, seed)).cuda().double()
    ls, lt = (torch.from_numpy(length[k]).cuda().long() for k in range(2))
    if case["gap"] == "log":
        w = torch.from_numpy(_gap(case).costs(max(case["s_hi"], case["t_hi"]) + 1)).cuda().double()
        best = _general(table[a.long()[:, :, None], b.long()[:, None, :]], ls, lt, w, case["locality"])
    else:
        b, k, flat = b.flip(1), case["letters"], table.flatten()
        nt = case["t_hi"]
        gap = ("linear", case["open"]) if case["gap"] == "linear" else ("affine", case["open"], case["extend"])

        def part(lo, hi):
            return _wavefront(lambda d, i0, i1: flat[(a[lo:hi, i0:i1] * k + b[lo:hi, nt - 1 - d + i0:nt - 1 - d + i1])
                                                     .long()], ls[lo:hi], lt[lo:hi], gap, case["locality"])
        best = torch.cat([part(lo, lo + 16384) for lo in range(0, case["pairs"], 16384)])
    second = "s_to_t" if kind == "module" else "maps"
    return {"scores": best, **({} if case["codomain"] == "score" else {second: None})}


def _exact_floats(case, seed):
    kind, B, n = case["kind"], case["pairs"], case["hi"]
    lengths = torch.from_numpy(_lengths(case, seed)).cuda()
    x = [v.double() for v in _floats(case, seed)]
    grad = case.get("grad", True)
    dtw = kind == "series"
    locality = case.get("locality", "global")
    gap = None if dtw else ("affine", float(np.float32(case["open"])), float(np.float32(case["extend"])))
    if grad:
        g = torch.Generator(device="cuda").manual_seed(seed + 1)
        up = (torch.rand(B, generator=g, device="cuda") + 0.5).double()
    if kind == "embed":
        e = [v / v.norm(dim=2, keepdim=True) for v in x]
    outs = []
    grads = [torch.zeros_like(v) for v in x] if grad else []
    dgap = [torch.zeros((), dtype=torch.float64, device="cuda") for _ in range(2)]
    chunk = max(1, int(2e9 / (n * n)))
    for lo in range(0, B, chunk):
        hi = min(B, lo + chunk)
        ls, lt = lengths[lo:hi, 0], lengths[lo:hi, 1]
        if dtw:
            X, Y = x[0][lo:hi], x[1][lo:hi].flip(1)
            diag = lambda d, i0, i1: -(X[:, i0:i1] - Y[:, n - 1 - d + i0:n - 1 - d + i1]).abs()  # noqa: E731
        else:
            if kind == "embed":  # the similarity is defined as the product of BF16 factors
                f0, f1 = (v[lo:hi].bfloat16().double() for v in e)
            S = x[0][lo:hi] if kind == "dense" else torch.bmm(f0, f1.transpose(1, 2))
            F = S.reshape(hi - lo, n * n)
            diag = lambda d, i0, i1: F[:, i0 * (n - 1) + d:(i1 - 1) * (n - 1) + d + 1:max(1, n - 1)]  # noqa: E731
        if not grad:
            outs.append(_wavefront(diag, ls, lt, gap, locality))
            continue
        best, codes, bi, bj = _wavefront(diag, ls, lt, gap, locality, codes=True)
        outs.append(-best if dtw else best)
        cells, opens, exts, ei, ej = _walk(codes, bi, bj, int(ls.max()), int(lt.max()), dtw)
        k, i, j = cells
        u = up[lo:hi]
        if dtw:
            s = torch.sign(x[0][lo + k, i] - x[1][lo + k, j]) * u[k]
            grads[0].index_put_((lo + k, i), s, accumulate=True)
            grads[1].index_put_((lo + k, j), -s, accumulate=True)
            continue
        if locality == "global":  # the gap that leads back to the corner
            rest = torch.maximum(ei, ej) + 1
            opens += (rest > 0).double()
            exts += (rest - 1).clamp_min(0).double()
        dgap[0] -= (opens * u).sum()
        dgap[1] -= (exts * u).sum()
        if kind == "dense":
            grads[0][lo + k, i, j] = u[k]
            continue
        es, et = e[0][lo + k, i], e[1][lo + k, j]
        cos = (es * et).sum(1, keepdim=True)
        grads[0][lo + k, i] = (et - cos * es) / x[0][lo + k, i].norm(dim=1, keepdim=True) * u[k][:, None]
        grads[1][lo + k, j] = (es - cos * et) / x[1][lo + k, j].norm(dim=1, keepdim=True) * u[k][:, None]
    scores = torch.cat(outs)
    if not grad:
        return {"scores": scores}
    return {"scores": scores, "grads": grads + ([] if dtw else dgap)}
