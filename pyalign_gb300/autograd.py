"""Differentiable optimal alignment scores (torch.autograd) on the GB300 kernels.

The reference has no gradients; this is the "differentiation" form of the batched solve.
The forward pass is the same sm_103a DP as the drop-in module (one optimal path per pair,
solver.h:2665-2705); the backward pass is the max-plus subgradient of the optimal score:
the indicator of the aligned cells of the optimal path for dScore/dS (every visited cell
for DTW) and the gap counts along the path for dScore/d(open, extend), computed by
`pa_path_gradients` from the paths the forward pass keeps on the device.  Gradients with
respect to embeddings flow through the similarity product by torch's autograd.

Tie-breaking follows the reference, so on inputs with ties the subgradient is the one of
the reference's optimal path.
"""

import ctypes
import functools
import threading
import types

import numpy as np
import torch

from . import algorithm as _alg

# A solver's buffers belong to the work queued on one stream by one thread, and so do the cached
# index arrays and the pinned buffer below: both are part of the keys.
_SOLVERS = {}
_lock = threading.Lock()  # around changes of the tables


class _Gap:
    def __init__(self, open_, extend):
        self.open, self.extend = float(open_), float(extend)

    def to_special_case(self):
        return {"affine": (self.open - self.extend, self.extend)}


class _Linear:
    def __init__(self, g):
        self.g = float(g)

    def to_special_case(self):
        return {"linear": self.g}


def _solver(batch, n_s, n_t, locality, direction, dtw, gap, stream=None):
    if stream is None:
        stream = torch.cuda.current_stream().cuda_stream
    key = (batch, n_s, n_t, locality, direction, dtw, gap, stream, threading.get_ident())
    s = _SOLVERS.get(key)
    if s is None:
        A = _alg
        d = {
            "solver": A.Type.DTW if dtw else A.Type.ALIGNMENT,
            "direction": A.Direction.__members__[direction.upper()],
            "batch": True, "batch_size": batch, "return_dup": False,
            "locality": A.Locality.__members__[locality.upper()],
            "codomain": types.SimpleNamespace(detail=A.Detail.ALIGNMENT, count=A.Count.ONE),
            "gap_cost": None if dtw else (_Linear(gap[0]) if gap[1] is None else _Gap(*gap)),
        }
        mod = A.m32 if max(n_s, n_t) >= 16000 else A.m16
        s = mod.create_solver(n_s, n_t, mod.create_options(d))
        with _lock:
            if len(_SOLVERS) > 32:
                _SOLVERS.clear()
            _SOLVERS[key] = s
    return s


def _lib():
    L = _alg.lib()
    if not getattr(L, "_pa_grad_bound", False):
        vp, i64, i32 = ctypes.c_void_p, ctypes.c_int64, ctypes.c_int32
        L.pa_solve_dense_paths.restype = i32
        L.pa_solve_dense_paths.argtypes = [vp, vp, vp, i64, i64, i64, i64, i64, vp, vp, vp, vp, vp]
        L.pa_dense_paths_work.restype = i64
        L.pa_dense_paths_work.argtypes = [vp, vp, i64, i64, i64, i64, i64, vp]
        L.pa_solve_dense_paths_work.restype = i32
        L.pa_solve_dense_paths_work.argtypes = L.pa_solve_dense_paths.argtypes + [i64, vp, i64]
        L.pa_solve_series_paths.restype = i32
        L.pa_solve_series_paths.argtypes = [vp, vp, i64, vp, i64, i64, i64, i64, vp, vp, vp, vp, vp]
        L.pa_path_gradients.restype = i32
        L.pa_path_gradients.argtypes = [i32, i32, i32, i64, vp, vp, vp, vp, vp, vp, i64, i64, vp, vp]
        L.pa_path_embedding_gradients.restype = i32
        L.pa_path_embedding_gradients.argtypes = [i64, i32, i32, vp, vp, vp, vp, vp, vp, vp, vp, vp, vp, i64, i64,
                                                  vp, vp, vp]
        L.pa_path_embedding_gradients_full.restype = i32
        L.pa_path_embedding_gradients_full.argtypes = L.pa_path_embedding_gradients.argtypes
        L.pa_normalize_rows_bf16.restype = i32
        L.pa_normalize_rows_bf16.argtypes = [vp, i64, i32, i32, vp, vp, vp]
        L.pa_normalize_rows_bf16_lengths.restype = i32
        L.pa_normalize_rows_bf16_lengths.argtypes = [vp, i64, i64, i32, i32, vp, vp, vp, vp]
        L.pa_normalize_rows_bf16_tiled.restype = i32
        L.pa_normalize_rows_bf16_tiled.argtypes = [vp, i64, i64, i32, i32, vp, i32, vp, vp, vp]
        L.pa_path_series_gradients.restype = i32
        L.pa_path_series_gradients.argtypes = [i64, vp, vp, vp, vp, vp, vp, i64, i64, vp, vp, vp]
        L.pa_similarity_bf16.restype = i32
        f32 = ctypes.c_float
        L.pa_similarity_bf16.argtypes = [vp, vp, i64, i64, i64, i32, vp, vp, vp, i64, vp, i64, i64, f32, f32, vp, vp]
        L.pa_similarity_rows.restype = i32
        L.pa_similarity_rows.argtypes = [vp, vp, i64, i64, i64, i32, i32, vp, vp, vp, i64, vp, i64, i64, vp, vp, vp, vp]
        L.pa_path_embedding_gradients_rows.restype = i32
        L.pa_path_embedding_gradients_rows.argtypes = [i64, i32, i32, vp, vp, vp, vp, vp, vp, vp, vp, i64, i64, vp, vp, vp]
        L.pa_pair_plan.restype = i32
        L.pa_pair_plan.argtypes = [vp, i32, i64, i64, i64, i32, i32, vp, vp, vp, vp]
        L.pa_content_hash.restype = ctypes.c_uint64
        L.pa_content_hash.argtypes = [vp, i64]
        L.pa_path_scores_f64.restype = i32
        L.pa_path_scores_f64.argtypes = [i32, i32, i32, i64, vp, vp, vp, vp, vp, i64, i64, vp, vp, vp, vp]
        L._pa_grad_bound = True
    return L


_STATUS = {}


def _status(device):
    st = _STATUS.get(device)
    if st is None:
        st = torch.zeros(1, dtype=torch.int32, device=device)
        _STATUS[device] = st
    return st


def tensor_core_status(device=None):
    """Error bits the tensor-core similarity kernel raised since the last call (2: a wait
    for the tensor cores timed out); reading synchronises the device and clears them."""
    st = _status(torch.device(device or "cuda", torch.cuda.current_device()))
    v = int(st.item())
    st.zero_()
    return v


_small_cache = {}   # (device, stream, dtype, shape, content hash) -> (host copy, device tensor): index arrays seen before
_staging = {}       # (thread, device, dtype) -> (pinned buffer, event of its last copy)


def _to_device(arr, device, stream=None):
    """A small host index array (lengths, offsets) on the device without blocking the host: a
    content-keyed cache (a training loop passes the same lengths every step; equal hashes are
    compared in full) and, for new contents, a non-blocking copy out of a reused pinned buffer.
    An array of one stream is not another's: its copy may still be queued there.  stream: the
    handle of the current one, if known."""
    arr = np.ascontiguousarray(arr)
    device = torch.device(device)
    if stream is None:
        stream = torch.cuda.current_stream(device).cuda_stream
    key = (str(device), stream, arr.dtype.str, arr.shape, _lib().pa_content_hash(arr.ctypes.data, arr.nbytes))
    hit = _small_cache.get(key)
    if hit is not None and np.array_equal(hit[0], arr):
        return hit[1]
    dtype = torch.from_numpy(arr[:0]).dtype
    mine = (threading.get_ident(), str(device), arr.dtype.str)
    buf, ev = _staging.get(mine, (None, None))
    if buf is None or buf.numel() < arr.size:
        buf, ev = torch.empty(max(arr.size, 1 << 14), dtype=dtype, pin_memory=True), None
    if ev is not None:
        ev.synchronize()  # the previous copy out of the buffer has finished
    flat = buf[:arr.size]
    flat.copy_(torch.from_numpy(arr.reshape(-1)))
    out = flat.to(device, non_blocking=True).reshape(arr.shape)
    ev = torch.cuda.Event()
    ev.record(torch.cuda.current_stream(device))
    with _lock:
        if mine not in _staging and len(_staging) >= 32:
            _staging.pop(next(iter(_staging)))
        _staging[mine] = (buf, ev)
        if key not in _small_cache and len(_small_cache) >= 32:
            _small_cache.pop(next(iter(_small_cache)))
        _small_cache[key] = (arr.copy(), out)
    return out


class _Plan:
    """The lengths of a batch of pairs as the calls below take them (pa_pair_plan, one pass on the
    host): ln (2, B) int32, meta = ln and the tile prefix of a product in tiles of SIM_TILE rows of
    s and tile_t rows of t, the packed path offsets, and the totals."""

    def __init__(self, lengths, B, n_s, n_t, what, tile_t=128):
        raw = np.asarray(lengths).reshape(B, 2)
        wide = raw.dtype == np.int64
        if not wide or not raw.flags.c_contiguous:
            raw, wide = np.ascontiguousarray(raw, dtype=np.int32), False
        self.meta = np.empty(3 * B + 1, np.int32)
        self.poff = np.empty(B, np.int64)
        self.ln = self.meta[:2 * B].reshape(2, B)
        tot = np.empty(2, np.int64)
        m = self.meta.ctypes.data
        if _lib().pa_pair_plan(raw.ctypes.data, int(wide), B, n_s, n_t, SIM_TILE, tile_t, m, m + 8 * B, self.poff.ctypes.data,
                               tot.ctypes.data):
            raise ValueError("lengths exceed " + what)
        self.tiles, self.entries = int(tot[0]), int(tot[1])


def _similarity_rows(Es, Et, lengths, normalize, out, plan=None):
    """S^T of <en_s, en_t> into out (batch, n_t, n_s) from float rows of a width that is a
    multiple of 4 up to ROWS_DIM (pa_similarity_rows), and 1 / |E| of the rows."""
    B, n_s, dim = Es.shape
    n_t = Et.shape[1]
    plan = plan or _Plan(lengths, B, n_s, n_t, "the embeddings", ROWS_TILE)
    stream = torch.cuda.current_stream().cuda_stream
    dmeta = _to_device(plan.meta, Es.device, stream)
    inv_s = torch.empty(B * n_s, dtype=torch.float32, device=Es.device)
    inv_t = torch.empty(B * n_t, dtype=torch.float32, device=Es.device)
    _alg.check(_lib().pa_similarity_rows(
        Es.data_ptr(), Et.data_ptr(), B, n_s, n_t, dim, int(normalize), dmeta.data_ptr(), dmeta.data_ptr() + 4 * B,
        dmeta.data_ptr() + 8 * B, plan.tiles, out.data_ptr(), out.stride(0), out.stride(1), inv_s.data_ptr(),
        inv_t.data_ptr(), _status(Es.device).data_ptr(), stream))
    return inv_s, inv_t


def similarity_bf16(Esb, Etb, lengths, out=None, alpha=1.0, beta=0.0):
    """S = beta + alpha <Es[i], Et[j]> per pair from BF16 factors (batch, n, dim), on the
    tensor cores (pa_similarity_bf16), FP32 accumulation (alpha = -1, beta = 1 gives the
    distance 1 - cos).  Only the cells inside each pair's lengths are written: the rest of
    `out` (a fresh torch.empty by default) is left as it was.  Returns S as a
    (batch, n_s, n_t) transposed view of S^T, stride 1 along s."""
    B, n_s, dim = Esb.shape
    n_t = Etb.shape[1]
    if Esb.dtype != torch.bfloat16 or Etb.dtype != torch.bfloat16 or not Esb.is_contiguous() \
            or not Etb.is_contiguous() or Etb.shape[0] != B or Etb.shape[2] != dim:
        raise ValueError("Es, Et must be contiguous BF16 (batch, n, dim) tensors of one batch and dim")
    if dim % 16:
        raise ValueError("dim must be a multiple of 16")
    plan = _Plan(lengths, B, n_s, n_t, "the embeddings")
    stream = torch.cuda.current_stream().cuda_stream
    dmeta, total = _to_device(plan.meta, Esb.device, stream), plan.tiles  # no host wait for the queued work
    if out is None:
        out = torch.empty((B, n_t, n_s), dtype=torch.float32, device=Esb.device)
    elif out.shape != (B, n_t, n_s) or out.dtype != torch.float32 or out.stride(2) != 1 or not out.is_cuda:
        raise ValueError("out must be a (batch, n_t, n_s) float32 CUDA tensor with unit stride along s")
    st = _status(Esb.device)
    _alg.check(_lib().pa_similarity_bf16(
        Esb.data_ptr(), Etb.data_ptr(), B, n_s, n_t, dim, dmeta.data_ptr(), dmeta.data_ptr() + 4 * B,
        dmeta.data_ptr() + 8 * B, total, out.data_ptr(), out.stride(0), out.stride(1), float(alpha), float(beta),
        st.data_ptr(), stream))
    return out.transpose(1, 2)


def _pad16(E):
    d = E.shape[-1]
    return E if d % 16 == 0 else torch.nn.functional.pad(E, (0, 16 - d % 16))


def path_scores_f64(S, lengths, gap_open=None, gap_extend=None, locality="global", direction="maximize",
                    dtw=False, with_scale=False):
    """The optimal scores of the float32 DP and, for the same recovered paths, their scores
    re-evaluated in FP64 on the GPU (pa_path_scores_f64): (scores float32, replay float64),
    plus with_scale the magnitude of the summed terms (sum |S| + gap costs) per path.  The
    distance between the two scores is the DP's float32 accumulation error."""
    linear = gap_extend is None
    gap = None if dtw else ((float(gap_open), None) if linear else (float(gap_open), float(gap_extend)))
    if S.stride(1) != 1 and S.stride(2) != 1:
        S = S.contiguous()
    scores, paths, plen, poff, _ = _forward_paths(S, lengths, gap, locality, direction, dtw)
    B = S.shape[0]
    A = _alg
    if dtw:
        g = None
    elif linear:
        g = np.array([gap[0], gap[0], gap[0], gap[0]], np.float64)
    else:
        g = np.array([gap[0], gap[1], gap[0], gap[1]], np.float64)
    soff = torch.from_numpy(S.storage_offset() + np.arange(B, dtype=np.int64) * S.stride(0)).to(S.device)
    base = S.data_ptr() - S.storage_offset() * S.element_size()
    out = torch.empty(B, dtype=torch.float64, device=S.device)
    scale = torch.empty(B, dtype=torch.float64, device=S.device) if with_scale else None
    _alg.check(_lib().pa_path_scores_f64(
        int(A.Type.DTW if dtw else A.Type.ALIGNMENT), int(A.Locality.__members__[locality.upper()]),
        int(A.Direction.__members__[direction.upper()]), B, paths.data_ptr(), poff.data_ptr(), plen.data_ptr(),
        base, soff.data_ptr(), S.stride(1), S.stride(2), None if g is None else g.ctypes.data, out.data_ptr(),
        None if scale is None else scale.data_ptr(), torch.cuda.current_stream().cuda_stream))
    return (scores, out, scale) if with_scale else (scores, out)


@functools.lru_cache(maxsize=32)
def _pair_offsets(B, first, stride):
    """Where the pairs' matrices begin (elements), as the host array a dense solve takes."""
    off = first + np.arange(B, dtype=np.int64) * stride
    off.flags.writeable = False
    return off


DENSE_ROOM_ASKED = 1 << 26  # bytes from which the room of a copy is worked out from the lengths


def _dense_work(S, args):
    """Room for a copy of S in the layout the DP reads fastest, from torch's allocator (which has it
    back for dS, of the same size): None where there is no room.  args: of pa_solve_dense_paths."""
    B, n_s, n_t = args[5:8]
    room = B * n_t * (n_s + 3 & ~3)
    if room > DENSE_ROOM_ASKED // 4:
        room = _lib().pa_dense_paths_work(*args[1:9]) // 4
    try:
        return S.new_empty(room) if room else None
    except torch.cuda.OutOfMemoryError:
        return None


def _forward_paths(S, lengths, gap, locality, direction, dtw, plan=None, rows=0):
    """Scores and optimal paths of the pairs of S (device); returns (scores, paths, path
    lengths, device path offsets, layout flag).  plan: the _Plan of the lengths if there is one; rows: entries
    of a column of S (stride 1 along s) that may be read, if more than its rows."""
    if not S.is_cuda or S.dtype != torch.float32 or S.dim() != 3:
        raise ValueError("S must be a (batch, len_s, len_t) float32 CUDA tensor")
    # any layout with unit stride along s or t is taken; a transposed view (stride 1 along s, rows
    # of whole 16-byte words) is the fastest, being read in place: others are copied to it first
    if S.stride(1) != 1 and S.stride(2) != 1:
        S = S.contiguous()
    B, n_s, n_t = S.shape
    ss, st_ = S.stride(1), S.stride(2)
    plan = plan or _Plan(lengths, B, n_s, n_t, "the similarity tensor")
    solver, ln, scores, paths, plen, poff, stream = _path_buffers(B, n_s, n_t, plan, locality, direction, dtw, gap, S.device)
    pair, first, ptr = S.stride(0), S.storage_offset(), S.data_ptr()
    offsets = _pair_offsets(B, first, pair)
    args = (solver.handle, ptr - 4 * first, offsets.ctypes.data, ss, st_, B, n_s, n_t, ln.ctypes.data,
            scores.data_ptr(), paths.data_ptr(), poff.ctypes.data, plen.data_ptr())
    L = _lib()
    # (these layouts are read in place, and room for a copy is ignored)
    in_place = ss == 1 and not (pair | st_) & 3 and not ptr & 15 and (n_s + 3 & ~3) <= max(n_s, rows)
    work = None if in_place else _dense_work(S, args)
    status = L.pa_solve_dense_paths_work(*args, rows, work.data_ptr() if work is not None else None,
                                         4 * work.numel() if work is not None else 0)
    if status and work is not None and "out of memory" in L.pa_last_error().decode():
        # the copy's room was the solver's last: without the copy
        del work
        torch.cuda.empty_cache()
        status = L.pa_solve_dense_paths(*args)
    _alg.check(status)
    return scores, paths, plen, _to_device(poff, S.device, stream), ss == 1


def _path_buffers(B, n_s, n_t, plan, locality, direction, dtw, gap, device):
    """The solver on the current stream, the (2, B) int32 lengths and the output buffers of a
    paths solve: scores, packed paths (2 (|s| + |t| + 2) entries per pair), path lengths and
    the host path offsets, and the stream's handle."""
    stream = torch.cuda.current_stream().cuda_stream
    solver = _solver(B, n_s, n_t, locality, direction, dtw, gap, stream)
    _alg.check(_lib().pa_solver_set_stream(solver.handle, ctypes.c_void_p(stream)))
    paths = torch.empty(plan.entries, dtype=torch.int32, device=device)
    plen = torch.zeros(B, dtype=torch.int32, device=device)
    scores = torch.empty(B, dtype=torch.float32, device=device)
    return solver, plan.ln, scores, paths, plen, plan.poff, stream


def _series_paths(x, y, lengths, gap, locality, direction, dtw):
    """_forward_paths for S(u, v) = |x_u - y_v| of the series rows of x and y (contiguous
    float32 CUDA tensors): the kernel computes each cell, no matrix is formed."""
    B, n_s = x.shape
    n_t = y.shape[1]
    plan = _Plan(lengths, B, n_s, n_t, "the series")
    solver, ln, scores, paths, plen, poff, stream = _path_buffers(B, n_s, n_t, plan, locality, direction, dtw, gap, x.device)
    _alg.check(_lib().pa_solve_series_paths(
        solver.handle, x.data_ptr(), x.stride(0), y.data_ptr(), y.stride(0), B, n_s, n_t, ln.ctypes.data,
        scores.data_ptr(), paths.data_ptr(), poff.ctypes.data, plen.data_ptr()))
    return scores, paths, plen, _to_device(poff, x.device, stream)


def _gap_grads(linear, locality, direction, B, paths, plen, poff, grad, device):
    """d score / d (open, extend) summed over pairs (pa_path_gradients without dS), on the gap
    costs' device (in one copy)."""
    A = _alg
    dgap = torch.empty((B, 4), dtype=torch.float32, device=grad.device)  # every pair writes its 4
    _alg.check(_lib().pa_path_gradients(
        int(A.Type.ALIGNMENT), int(A.Locality.__members__[locality.upper()]),
        int(A.Direction.__members__[direction.upper()]), B, paths.data_ptr(), poff.data_ptr(),
        plen.data_ptr(), grad.data_ptr(), None, None, 0, 0, dgap.data_ptr(),
        torch.cuda.current_stream().cuda_stream))
    # one reduction: (open_s + open_t, extend_s + extend_t) summed over pairs
    if linear:
        return dgap.sum(), None
    tot = dgap.view(B, 2, 2).sum(dim=(0, 1)).to(device)
    return tot[0], tot[1]


class AlignmentScore(torch.autograd.Function):
    """Optimal alignment score of each pair; backward = path indicator and gap counts."""

    @staticmethod
    def forward(ctx, S, lengths, gap_open, gap_extend, locality, direction, dtw, linear):
        gap = None if dtw else ((float(gap_open), None) if linear else (float(gap_open), float(gap_extend)))
        scores, paths, plen, poff, transposed = _forward_paths(S, lengths, gap, locality, direction, dtw)
        ctx.save_for_backward(paths, plen, poff)
        ctx.meta = (S.shape, locality, direction, dtw, linear, transposed, gap_open.device)
        return scores

    @staticmethod
    def backward(ctx, grad):
        paths, plen, poff = ctx.saved_tensors
        (B, n_s, n_t), locality, direction, dtw, linear, transposed, gap_device = ctx.meta
        A = _alg
        grad = grad.contiguous().float()
        # dS in the layout S came in: a transposed view when S was one
        if transposed:
            dS = torch.zeros((B, n_t, n_s), dtype=torch.float32, device=grad.device).transpose(1, 2)
        else:
            dS = torch.zeros((B, n_s, n_t), dtype=torch.float32, device=grad.device)
        dgap = torch.empty((B, 4), dtype=torch.float32, device=grad.device)  # every pair writes its 4
        offsets = torch.arange(B, dtype=torch.int64, device=grad.device) * (n_s * n_t)
        _alg.check(_lib().pa_path_gradients(
            int(A.Type.DTW if dtw else A.Type.ALIGNMENT), int(A.Locality.__members__[locality.upper()]),
            int(A.Direction.__members__[direction.upper()]), B, paths.data_ptr(), poff.data_ptr(),
            plen.data_ptr(), grad.data_ptr(), dS.data_ptr(), offsets.data_ptr(), dS.stride(1), dS.stride(2),
            dgap.data_ptr(), torch.cuda.current_stream().cuda_stream))
        if dtw or not any(ctx.needs_input_grad[2:4]):
            return dS, None, None, None, None, None, None, None
        tot = dgap.sum(dim=0).to(gap_device)  # in one copy
        if linear:
            d_open, d_ext = tot[0] + tot[1] + tot[2] + tot[3], None
        else:
            d_open, d_ext = tot[0] + tot[2], tot[1] + tot[3]
        return dS, None, d_open, d_ext, None, None, None, None


def alignment_score(S, lengths, gap_open=None, gap_extend=None, locality="global", direction="maximize",
                    dtw=False):
    """Differentiable optimal scores of `batch` pairs.

    S: (batch, len_s, len_t) float32 CUDA tensor of similarities (distances when
    minimizing), padded; lengths: (batch, 2) of |s|, |t|.  Affine gaps w(k) = open +
    extend (k - 1) when both are given, linear w(k) = open * k when gap_extend is None;
    DTW ignores gaps.  gap_open/gap_extend may be tensors that require grad.
    """
    linear = gap_extend is None
    go = gap_open if isinstance(gap_open, torch.Tensor) else torch.tensor(float(gap_open or 0.0))
    ge = gap_extend if isinstance(gap_extend, torch.Tensor) else torch.tensor(float(gap_extend or 0.0))
    return AlignmentScore.apply(S, lengths, go, ge, locality, direction, dtw, linear)


SIM_TILE = 128  # rows of a tile of the tensor-core product (pa_simgemm.cu TM, TN)
ROWS_TILE = 256  # rows of t of a tile of the product from float rows, and its largest width (FB, FDIM)
ROWS_DIM = 256
ROWS_MARKS = 190000  # rows of s and t whose marks fit the backward's shared memory


def normalized_bf16(E, normalize=True, lengths=None, tiled=False):
    """The BF16 factor of E (batch, n, d) for the similarity product -- E / |E| per row when
    normalising -- and 1 / |E| per row, in one pass (pa_normalize_rows_bf16).  d is padded
    with zeros to a multiple of 16 (the tensor-core K step).  With ``lengths`` (batch,) the
    rows past each pair's length are zero and not read (pa_normalize_rows_bf16_lengths);
    with ``tiled`` only the rows the product's tiles read are written (up to each length
    rounded up to SIM_TILE; the rows beyond keep whatever the fresh tensor held), for a factor
    that only similarity_bf16 and the aligned rows of the backward read."""
    E = _pad16(E.contiguous().float())
    B, n, dim = E.shape
    Eb = torch.empty(E.shape, dtype=torch.bfloat16, device=E.device)
    inv = torch.empty(B * n, dtype=torch.float32, device=E.device)
    stream = torch.cuda.current_stream().cuda_stream
    if lengths is None:
        _alg.check(_lib().pa_normalize_rows_bf16(E.data_ptr(), B * n, dim, int(normalize), Eb.data_ptr(),
                                                 inv.data_ptr(), stream))
    else:
        ln = _to_device(np.minimum(np.asarray(lengths).reshape(B), n).astype(np.int32), E.device, stream)
        if tiled:
            _alg.check(_lib().pa_normalize_rows_bf16_tiled(E.data_ptr(), B, n, dim, int(normalize), ln.data_ptr(),
                                                           SIM_TILE, Eb.data_ptr(), inv.data_ptr(), stream))
        else:
            _alg.check(_lib().pa_normalize_rows_bf16_lengths(E.data_ptr(), B, n, dim, int(normalize),
                                                             ln.data_ptr(), Eb.data_ptr(), inv.data_ptr(), stream))
    return Eb, inv


class CosineSimilarity(torch.autograd.Function):
    """S = <en_s, en_t> with en = E / |E|, the product on the tensor cores.  Backward: the
    dense route, dEn_s = dS en_t and dEn_t = dS^T en_s (the BF16 cast passes gradients
    through), then the normalisation backward (g - (g . en) en) / |E|."""

    @staticmethod
    def forward(ctx, Es, Et, lengths):
        B, n_s, d = Es.shape
        n_t = Et.shape[1]
        ln = None if lengths is None else np.asarray(lengths).reshape(B, 2)
        Esb, inv_s = normalized_bf16(Es, True, None if ln is None else ln[:, 0])  # padding rows: zero
        Etb, inv_t = normalized_bf16(Et, True, None if ln is None else ln[:, 1])
        if lengths is None:
            lengths = np.tile(np.array([[n_s, n_t]], np.int32), (B, 1))
            out = None
        else:
            out = torch.zeros((B, n_t, n_s), dtype=torch.float32, device=Es.device)
        ctx.save_for_backward(Esb, Etb, inv_s, inv_t)
        ctx.d = d
        return similarity_bf16(Esb, Etb, lengths, out=out)

    @staticmethod
    def backward(ctx, dS):
        Esb, Etb, inv_s, inv_t = ctx.saved_tensors
        B, n_s, dp = Esb.shape
        n_t = Etb.shape[1]
        en_s, en_t = Esb.float(), Etb.float()
        g_s = torch.bmm(dS.float(), en_t)
        g_t = torch.bmm(dS.float().transpose(1, 2), en_s)
        inv_s = inv_s.view(B, n_s, 1)
        inv_t = inv_t.view(B, n_t, 1)
        # en here is the BF16 factor; the normalisation backward uses the exact en = E / |E|
        # only through (g . en) en, where the BF16 rounding is below float32 noise of g
        d_s = (g_s - (g_s * en_s).sum(-1, keepdim=True) * en_s) * inv_s
        d_t = (g_t - (g_t * en_t).sum(-1, keepdim=True) * en_t) * inv_t
        return d_s[..., :ctx.d], d_t[..., :ctx.d], None


def cosine_similarity_batch(Es, Et, lengths=None):
    """S = cos(E_s, E_t) per pair: L2-normalised embeddings multiplied in BF16 with FP32
    accumulation on the tensor cores.  Es: (batch, len_s, d), Et: (batch, len_t, d);
    lengths (batch, 2) limits the product to each pair's cells (the rest of S is zero).
    Returned as a transposed view of S^T (stride 1 along s), the layout the DP reads
    fastest.  Differentiable with respect to Es and Et."""
    return CosineSimilarity.apply(Es, Et, lengths)


class EmbeddingAlignmentScore(torch.autograd.Function):
    """Alignment score of S = <en_s, en_t^T> for per-token embeddings (en = E/|E| for the
    cosine, E for the dot product), the product in BF16 with FP32 accumulation.  The
    backward walks the optimal paths and writes the gradients of the aligned rows of E
    directly, through the normalisation (pa_path_embedding_gradients): O(path * d) work
    instead of a dense dS, two batched products and a dense normalisation backward."""

    @staticmethod
    def forward(ctx, Es, Et, lengths, gap_open, gap_extend, locality, direction, linear, normalize):
        if Es.dim() != 3 or Et.dim() != 3 or not Es.is_cuda or Et.device != Es.device:
            raise ValueError("Es, Et must be (batch, len, d) CUDA tensors on one device")
        dim_in = Es.shape[-1]
        Es, Et = Es.contiguous().float(), Et.contiguous().float()
        # the product straight from the float rows where their width allows it; else through stored
        # BF16 factors, of widths padded to the tensor cores' K step
        rows = dim_in % 4 == 0 and 0 < dim_in <= ROWS_DIM and Es.shape[1] + Et.shape[1] <= ROWS_MARKS \
            and Et.shape[0] == Es.shape[0] and Et.shape[2] == dim_in and (Es.data_ptr() | Et.data_ptr()) % 16 == 0
        Esb = Etb = None
        if not rows:
            Es, Et = _pad16(Es), _pad16(Et)
            ln = np.asarray(lengths).reshape(Es.shape[0], 2)
            # rows past a pair's length: zero up to the product's tile, not read, not written beyond
            Esb, inv_s = normalized_bf16(Es, normalize, ln[:, 0], tiled=True)
            Etb, inv_t = normalized_bf16(Et, normalize, ln[:, 1], tiled=True)
        # S^T = en_t en_s^T on the tensor cores, only the cells inside the lengths; its
        # transposed view is S with stride 1 along s; its columns are padded to whole 16-byte
        # words for the DP's loads (the solver keeps the true number of rows, on which the
        # rounding of its border costs depends)
        B, n_s, n_t = Es.shape[0], Es.shape[1], Et.shape[1]
        St = torch.empty((B, n_t, n_s + 3 & ~3), dtype=torch.float32, device=Es.device)
        plan = None
        if rows:
            plan = _Plan(lengths, B, n_s, n_t, "the embeddings", ROWS_TILE)
            inv_s, inv_t = _similarity_rows(Es, Et, lengths, normalize, St, plan)
        else:
            similarity_bf16(Esb, Etb, lengths, out=St[:, :, :n_s])
        pitch = St.shape[2]
        S = St.transpose(1, 2) if pitch == n_s else St.transpose(1, 2).narrow(1, 0, n_s)
        gap = (float(gap_open), None) if linear else (float(gap_open), float(gap_extend))
        scores, paths, plen, poff, _ = _forward_paths(S, lengths, gap, locality, direction, False, plan, pitch)
        ctx.save_for_backward(Es, Et, Esb, Etb, inv_s, inv_t, paths, plen, poff)
        ctx.meta = (locality, direction, linear, normalize, gap_open.device)
        ctx.dim_in = dim_in
        return scores

    @staticmethod
    def backward(ctx, grad):
        Es, Et, Esb, Etb, inv_s, inv_t, paths, plen, poff = ctx.saved_tensors
        locality, direction, linear, normalize, gap_device = ctx.meta
        grad = grad.contiguous().float()
        B, n_s, dim = Es.shape
        n_t = Et.shape[1]
        d_in = ctx.dim_in
        dEs = torch.empty_like(Es)  # every row is written: the aligned ones, zeros elsewhere
        dEt = torch.empty_like(Et)
        walk = (B, dim, int(normalize), paths.data_ptr(), poff.data_ptr(), plen.data_ptr(), grad.data_ptr(),
                Es.data_ptr(), Et.data_ptr())
        out = (inv_s.data_ptr(), inv_t.data_ptr(), n_s, n_t, dEs.data_ptr(), dEt.data_ptr(),
               torch.cuda.current_stream().cuda_stream)
        if Esb is None:
            _alg.check(_lib().pa_path_embedding_gradients_rows(*walk, *out))
        else:
            _alg.check(_lib().pa_path_embedding_gradients_full(*walk, Esb.data_ptr(), Etb.data_ptr(), *out))
        d_open = d_ext = None
        if any(ctx.needs_input_grad[3:5]):
            d_open, d_ext = _gap_grads(linear, locality, direction, B, paths, plen, poff, grad, gap_device)
        return dEs[..., :d_in], dEt[..., :d_in], None, d_open, d_ext, None, None, None, None


def embedding_alignment_score(Es, Et, lengths, gap_open, gap_extend=None, locality="global",
                              direction="maximize", normalize=True):
    """Differentiable alignment scores on the cosine (normalize=True) or dot similarity of
    per-token embeddings Es (batch, len_s, d) and Et (batch, len_t, d), padded."""
    linear = gap_extend is None
    go = gap_open if isinstance(gap_open, torch.Tensor) else torch.tensor(float(gap_open))
    ge = gap_extend if isinstance(gap_extend, torch.Tensor) else torch.tensor(float(gap_extend or 0.0))
    return EmbeddingAlignmentScore.apply(Es, Et, lengths, go, ge, locality, direction, linear, normalize)


class SeriesDTW(torch.autograd.Function):
    """DTW score (minimize) of series pairs with d(u, v) = |x_u - y_v|; the backward walks
    the optimal paths (pa_path_series_gradients)."""

    @staticmethod
    def forward(ctx, x, y, lengths):
        x = x.contiguous().float()
        y = y.contiguous().float()
        if x.dim() != 2 or y.dim() != 2 or x.shape[0] != y.shape[0] or not x.is_cuda or y.device != x.device:
            raise ValueError("x, y must be (batch, len) CUDA tensors on one device")
        scores, paths, plen, poff = _series_paths(x, y, lengths, None, "global", "minimize", True)
        ctx.save_for_backward(x, y, paths, plen, poff)
        return scores

    @staticmethod
    def backward(ctx, grad):
        x, y, paths, plen, poff = ctx.saved_tensors
        grad = grad.contiguous().float()
        dx = torch.zeros_like(x)
        dy = torch.zeros_like(y)
        _alg.check(_lib().pa_path_series_gradients(
            x.shape[0], paths.data_ptr(), poff.data_ptr(), plen.data_ptr(), grad.data_ptr(), x.data_ptr(),
            y.data_ptr(), x.shape[1], y.shape[1], dx.data_ptr(), dy.data_ptr(),
            torch.cuda.current_stream().cuda_stream))
        return dx, dy, None


def dtw_series_score(x, y, lengths):
    """Differentiable DTW (minimize, |x_u - y_v|) of series x (batch, len_s), y (batch, len_t)."""
    return SeriesDTW.apply(x, y, lengths)
