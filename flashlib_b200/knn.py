"""Fused exact brute-force kNN behind flashlib's ``flash_knn`` signature.

Mirrors ``flashlib/primitives/knn/impl.py:199-287`` (``flash_knn_dispatch``): same
arguments, same return dtypes on CUDA (``vals`` fp32 true squared L2, ``idxs`` int32),
same error behaviour for unknown backends.  The reference's multi-backend routing is
gone: every call goes through the C ABI into the sm_100a kernels, and CPU tensors are
rejected because this library has no CPU path.
"""
from __future__ import annotations

import ctypes
import os
import time
import weakref
from collections import OrderedDict, deque
from typing import Optional

import torch

from . import _lib

_VALID_BACKENDS = ("triton", "cutedsl", "torch")
_MODES = {None: _lib.FL_KNN_AUTO, "auto": _lib.FL_KNN_AUTO, "exact": _lib.FL_KNN_EXACT_SIMT,
          "simt": _lib.FL_KNN_EXACT_SIMT, "bf16": _lib.FL_KNN_BF16_RERANK,
          "tc": _lib.FL_KNN_BF16_RERANK}


_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def _stream_ptr(device: torch.device) -> int:
    if _raw_stream is not None and device.index is not None:
        return _raw_stream(device.index)       # the handle alone, without building a Stream object
    return torch.cuda.current_stream(device).cuda_stream


_STREAMS: dict = {}


def _stream(device: torch.device) -> torch.cuda.Stream:
    """The current stream as an object (building one takes 2 us; they are kept by handle)."""
    key = (device.index, _stream_ptr(device))
    hit = _STREAMS.get(key)
    if hit is None:
        if len(_STREAMS) >= 64:
            _STREAMS.clear()
        hit = _STREAMS[key] = torch.cuda.current_stream(device)
    return hit


class _OnDevice:
    """``torch.cuda.device`` for the (usual) case that the tensor's device is current already: no
    context is entered then."""

    __slots__ = ("_ctx",)

    def __init__(self, device: torch.device):
        self._ctx = None if device.index == torch.cuda.current_device() else torch.cuda.device(device)

    def __enter__(self):
        if self._ctx is not None:
            self._ctx.__enter__()

    def __exit__(self, *exc):
        if self._ctx is not None:
            self._ctx.__exit__(*exc)


def _capture_id(device: torch.device) -> int:
    """Number of the graph capture the current stream takes part in (0: none)."""
    return _lib.load().fl_stream_capture_id(_stream_ptr(device)) if torch.cuda.is_current_stream_capturing() else 0


def _nothing():
    return None


class _Built:
    """Where a kept buffer was filled.  Work on another stream is not ordered behind that: ``join`` makes the current
    stream wait for it and tells the allocator that this stream reads the buffer, which may leave its cache
    meanwhile.  A buffer filled under capture holds nothing until the graph runs, and only that graph may use it."""

    __slots__ = ("device", "stream", "capture", "event")

    def __init__(self, device: torch.device):
        self.device = device
        self.stream = _stream_ptr(device)
        self.capture = _capture_id(device)
        self.event = torch.cuda.Event()
        self.event.record(_stream(device))

    def __reduce__(self):
        return _nothing, ()            # a copy of an index or its pickle carries no event

    def usable(self) -> bool:
        return self.capture == 0 or self.capture == _capture_id(self.device)

    def join(self, buf: torch.Tensor) -> None:
        if _stream_ptr(self.device) == self.stream:
            return
        if _capture_id(self.device) != self.capture:
            return           # a capture may not wait for work outside it; torch.cuda.graph waits for the device first
        cur = _stream(self.device)
        cur.wait_event(self.event)
        buf.record_stream(cur)


# Entries that a graph was captured with: their addresses are in it, so they stay although their cache
# drops them, until the rows they stand for are freed.
_IN_GRAPHS: dict = {}


def _keep_for_graph(key, entry, t: torch.Tensor) -> None:
    if torch.cuda.is_current_stream_capturing() and _IN_GRAPHS.get(key) is not entry:
        if key not in _IN_GRAPHS:
            _evict_when_freed(_IN_GRAPHS, key, t)
        _IN_GRAPHS[key] = entry


def _as_f32_rows(t: torch.Tensor) -> torch.Tensor:
    """fp32 tensor whose last dimension is contiguous (rows may be strided)."""
    if t.dtype != torch.float32:
        t = t.float()
    if t.stride(-1) != 1 or (t.dim() == 2 and t.stride(0) < t.shape[1]):
        t = t.contiguous()
    return t


_DTYPE_CODES = {torch.float32: _lib.FL_DTYPE_F32, torch.bfloat16: _lib.FL_DTYPE_BF16, torch.float16: _lib.FL_DTYPE_F16}


def _as_rows(t: torch.Tensor) -> torch.Tensor:
    """Rows the kernels read as they are: fp32, bf16 or fp16 (anything else is converted to fp32),
    last dimension contiguous."""
    if t.dtype not in _DTYPE_CODES:
        t = t.float()
    if t.stride(-1) != 1 or (t.dim() == 2 and t.stride(0) < t.shape[1]):
        t = t.contiguous()
    return t


# Restatement of the reference's tol -> storage dtype rule (flashlib/linalg/gemm/__init__.py:114-207):
# among the GEMM variants whose declared residual is <= tol the one with the highest listed throughput
# is chosen, and only "fp16" / "bf16" name a storage dtype.  fp16 (residual 4e-4, 892 TF) beats bf16
# (3e-3, 816 TF) whenever both qualify, and tf32 (3e-4, 386 TF) qualifies alone below 4e-4.
_TOL_VARIANTS = (("fp16", 4e-4, 892.0, torch.float16), ("bf16", 3e-3, 816.0, torch.bfloat16), ("tf32", 3e-4, 386.0, None))


def storage_dtype_for(tol: Optional[float]):
    """16-bit dtype the inputs may be stored in for this ``tol`` (``None``: keep them as given)."""
    if tol is None or tol <= 0:
        return None
    ok = [v for v in _TOL_VARIANTS if v[1] <= tol]
    if not ok:
        return None
    return max(ok, key=lambda v: v[2])[3]


_CAST_CACHE: "OrderedDict[tuple, tuple]" = OrderedDict()       # key -> (16-bit rows, where they were written)


def _cast_rows_cached(c: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
    """``c.to(dtype)``, kept while ``c`` is alive and unchanged: the database is stored in 16 bits once,
    and its operand plane is found again on the next call."""
    key = _plane_key(c) + (dtype,)
    hit = _CAST_CACHE.get(key)
    if hit is not None and hit[1].usable():
        _CAST_CACHE[key] = hit
        _CAST_CACHE.move_to_end(key)
        hit[1].join(hit[0])
        _keep_for_graph(key, hit, c)
        return hit[0]
    out = c.to(dtype)
    entry = _CAST_CACHE[key] = (out, _Built(c.device))
    _evict_when_freed(_CAST_CACHE, key, c)
    _keep_for_graph(key, entry, c)
    while len(_CAST_CACHE) > _PLANE_CACHE_SIZE:
        _CAST_CACHE.popitem(last=False)
    return out


def _mode_from(mode: Optional[str]) -> int:
    if mode is None:
        mode = os.environ.get("FLASHLIB_B200_KNN_MODE") or None
    if mode not in _MODES:
        raise ValueError(f"mode must be one of {sorted(k for k in _MODES if k)} or None, got {mode!r}")
    return _MODES[mode]


class DbPlane:
    """The bf16 operand plane (+ half norms) of one database, built once per database and kept for the four last used
    (``clear_plane_cache`` gives them back): 2 bytes per feature, padded to 64, and 36 per row.

    The reference caches ``||c||^2`` per ``data_ptr`` in the same spirit
    (``flashlib/primitives/knn/triton/_row_norm.py:82-93``).
    """

    def __init__(self, db: torch.Tensor):
        lib = _lib.load()
        m, d = db.shape
        nbytes = lib.fl_knn_plane_bytes(m, d)
        self.buf = torch.empty(nbytes, dtype=torch.uint8, device=db.device)
        _lib.check(lib.fl_knn_prepare_db_rows(db.data_ptr(), _DTYPE_CODES[db.dtype], m, d, db.stride(0),
                                              self.buf.data_ptr(), nbytes, _stream_ptr(db.device)))
        self.key = _plane_key(db)
        self.built = _Built(db.device)
        self.split = None              # (buffer, where it was filled); False: none for this database

    @property
    def ptr(self) -> int:
        """Address of the plane, for a call on the current stream."""
        self.built.join(self.buf)
        return self.buf.data_ptr()

    def split_ptr(self, db: torch.Tensor):
        """Address of the split (hi/lo bf16) plane of the same database, built on first use; ``None``
        when the shape has none (d > 128) or it would exceed the size limit."""
        split = self.split
        if split is None or (split is not False and not split[1].usable()):
            lib = _lib.load()
            m, d = db.shape
            nbytes = lib.fl_knn_split_plane_bytes(m, d) if db.dtype == torch.float32 else 0
            if nbytes == 0 or nbytes > _split_plane_limit():
                split = False
            else:
                buf = torch.empty(nbytes, dtype=torch.uint8, device=db.device)
                _lib.check(lib.fl_knn_prepare_split_f32(db.data_ptr(), m, d, db.stride(0), buf.data_ptr(),
                                                        nbytes, _stream_ptr(db.device)))
                built = self.built
                if built.stream == _stream_ptr(db.device) and built.capture == _capture_id(db.device):
                    built.event.record(_stream(db.device))      # one event for the two of them
                else:
                    built = _Built(db.device)
                split = (buf, built)
            self.split = split             # (only now: another thread must not meet a plane nobody has enqueued yet)
        if split is False:
            return None
        split[1].join(split[0])
        return split[0].data_ptr()


def _split_plane_limit() -> int:
    """Largest split plane (bytes) built without being asked for: it takes 6.25x the fp32 rows'
    memory at d = 128 -> on for databases of a few million rows, off for the 100M-row shards."""
    return int(os.environ.get("FLASHLIB_B200_SPLIT_MAX_MB", "4096")) << 20


def _second_stage_default() -> bool:
    return os.environ.get("FLASHLIB_B200_KNN_STAGE2", "1") != "0"


def _plane_key(db: torch.Tensor):
    return (db.data_ptr(), tuple(db.shape), db.stride(0), db._version, db.device.index, db.dtype)


def _evict_when_freed(cache, key, t: torch.Tensor) -> None:
    """Drops ``cache[key]`` when the tensor that owns ``t``'s memory dies: a later tensor can
    be given the same address, shape and version, and must not meet the old entry."""
    owner = t._base if t._base is not None else t
    weakref.finalize(owner, cache.pop, key, None)


_PLANE_CACHE: "OrderedDict[tuple, DbPlane]" = OrderedDict()
_PLANE_CACHE_SIZE = 4


def get_plane(db: torch.Tensor) -> DbPlane:
    key = _plane_key(db)
    hit = _PLANE_CACHE.get(key)
    if hit is not None and hit.built.usable():
        _PLANE_CACHE[key] = hit            # (another thread may have dropped it since)
        _PLANE_CACHE.move_to_end(key)
        _keep_for_graph(key, hit, db)
        return hit
    plane = DbPlane(db)
    _PLANE_CACHE[key] = plane
    _evict_when_freed(_PLANE_CACHE, key, db)
    _keep_for_graph(key, plane, db)
    while len(_PLANE_CACHE) > _PLANE_CACHE_SIZE:
        _PLANE_CACHE.popitem(last=False)
    return plane


def clear_plane_cache() -> None:
    _PLANE_CACHE.clear()


# Status words of calls whose check was deferred.  The tensor-core kernels report a timed-out wait
# there; reading them right after the call would serialise host and device once per call, so the
# public entry points look at the words of EARLIER calls instead (and ``check_pending()`` looks at
# all of them).  A slot is a few words of pinned host memory that the last kernel of a call fills in,
# completion mark last: neither a copy nor an event enters the stream.  A call that is captured into a graph
# takes none: every replay would write to the slot, whosever it is by then.
class _StatusSlot:
    __slots__ = ("buf", "words", "ptr", "device")

    def __init__(self, device: torch.device):
        self.buf = torch.zeros(_lib.FL_STATUS_WORDS + 1, dtype=torch.int32).pin_memory()
        self.ptr = self.buf.data_ptr()
        self.words = (ctypes.c_int32 * (_lib.FL_STATUS_WORDS + 1)).from_address(self.ptr)
        self.device = device


_PENDING_STATUS: deque = deque()
_FREE_SLOTS: deque = deque()               # at most as many as calls were pending at once (64)


def _take_status_slot(device: torch.device) -> _StatusSlot:
    check_pending(block=False)
    while len(_PENDING_STATUS) >= 64:      # bounded: the oldest calls have long finished
        _finish_slot(_PENDING_STATUS.popleft(), wait=True)
    try:
        slot = _FREE_SLOTS.popleft()
    except IndexError:
        slot = _StatusSlot(device)
    slot.device = device
    slot.words[_lib.FL_STATUS_WORDS] = 0
    return slot


def _finish_slot(slot: _StatusSlot, wait: bool) -> bool:
    """Looks at a slot's words (waiting for its call first when asked to) and gives the slot back;
    ``False`` when the call is still running."""
    if slot.words[_lib.FL_STATUS_WORDS] == 0:
        if not wait:
            return False
        _await_mark(slot)
    st = list(slot.words)[:_lib.FL_STATUS_WORDS]
    _FREE_SLOTS.append(slot)
    _raise_on_status(st)
    return True


def _await_mark(slot: _StatusSlot) -> None:
    """Waits for this slot's own call and for nothing else on the device."""
    look = time.monotonic() + 1.0
    while slot.words[_lib.FL_STATUS_WORDS] == 0:
        time.sleep(2e-5)
        if time.monotonic() >= look:       # a device that has failed writes no mark: the query raises then
            torch.cuda.current_stream(slot.device).query()
            look += 1.0


_STATUS_TEXT = {_lib.FL_ETIMEOUT: "a bounded device-side wait ran out",
                _lib.FL_EUNSUPPORTED: "the call ran with timing-experiment flags set",
                _lib.FL_EWORKSPACE: "the fallback list overflowed"}


def _raise_on_status(st) -> None:
    err = st[_lib.FL_STATUS_ERROR]
    if err != 0:
        raise _lib.FlashlibError(
            f"tensor-core kernel reported status {err} ({_STATUS_TEXT.get(err, 'unknown')}; "
            f"where={st[_lib.FL_STATUS_WHERE]:#x}): the results of that call are invalid")


def check_pending(block: bool = True) -> None:
    """Raises if an earlier call whose status check was deferred reported an error.  With
    ``block=False`` only calls that have already finished on the device are looked at."""
    while _PENDING_STATUS:
        try:
            slot = _PENDING_STATUS.popleft()
        except IndexError:                 # another thread took it
            return
        if not block and slot.words[_lib.FL_STATUS_WORDS] == 0:
            _PENDING_STATUS.appendleft(slot)
            return
        _finish_slot(slot, wait=True)


def _defer_status_check(status: torch.Tensor) -> None:
    """Queues the status words of a call that has just been launched on the current stream."""
    if torch.cuda.is_current_stream_capturing():
        return
    slot = _take_status_slot(status.device)
    _lib.check(_lib.load().fl_publish_status(status.data_ptr(), slot.ptr, _stream_ptr(status.device)))
    _PENDING_STATUS.append(slot)


# Which kernel a shape takes and the workspace it needs: asked from the library once per device and shape.
_PLANS: dict = {}


def _knn_plan(lib, dev: Optional[int], nq: int, m: int, d: int, k: int, mode: int):
    """``(resolved mode, mode to pass on, wants an operand plane, workspace bytes, staged workspace bytes)``."""
    key = (dev, nq, m, d, k, mode)
    hit = _PLANS.get(key)
    if hit is not None:
        return hit
    resolved = lib.fl_knn_resolve_mode(nq, m, d, k) if mode == _lib.FL_KNN_AUTO else mode
    wants = resolved == _lib.FL_KNN_BF16_RERANK
    passed = resolved
    if not wants and mode == _lib.FL_KNN_AUTO and nq > 0 and lib.fl_knn_wants_plane(nq, m, d, k):
        # more than 512 features: automatic mode with a plane takes the streamed tensor-core kernel
        resolved, passed, wants = _lib.FL_KNN_BF16_RERANK, _lib.FL_KNN_AUTO, True
    ws = lib.fl_knn_workspace_bytes(max(nq, 1), m, d, k, passed)
    staged = lib.fl_knn_staged_workspace_bytes(nq, m, d, k) if passed == _lib.FL_KNN_BF16_RERANK else 0
    if len(_PLANS) >= 512:
        _PLANS.clear()
    plan = _PLANS[key] = (resolved, passed, wants, ws, staged)
    return plan


def knn_f32(q: torch.Tensor, db: torch.Tensor, k: int, *, mode: int = _lib.FL_KNN_AUTO,
            row_offset: int = 0, plane: Optional[DbPlane] = None, check_status=True,
            second_stage: Optional[bool] = None, out=None):
    """One 2-D problem through ``fl_knn_search`` (fp32, or bf16 / fp16 rows read as stored): returns
    ``(dist fp32 (nq,k), idx int32 (nq,k), info)``, in ``out = (dist, idx)`` when given.
    ``check_status=True`` reads the kernel's status words before returning (one host/device
    round trip; ``info["fallback_rows"]`` and ``info["stage2_rows"]`` are filled), ``"deferred"``
    leaves that to a later call or to ``check_pending()``, ``False`` skips it (so does ``"deferred"`` while
    the stream is captured: nobody reads the words of a replay).
    ``second_stage`` (tensor-core mode): rows the bf16 proof rejects are scored again on the
    tensor cores with split hi/lo operands before anything takes the exact CUDA-core pass;
    ``None`` = when the database's split plane exists or is small enough to build."""
    lib = _lib.load()
    nq, d = q.shape
    m = db.shape[0]
    dev = q.device
    _lib.require_device(dev.index)
    if q.dtype != db.dtype or db.dtype not in _DTYPE_CODES:
        raise TypeError(f"knn_f32 takes q and db of one dtype out of fp32 / bf16 / fp16, got {q.dtype} and {db.dtype}")
    resolved, passed, wants_plane, ws_bytes, staged_bytes = _knn_plan(lib, dev.index, nq, m, d, k, mode)
    if wants_plane and plane is None:
        try:
            plane = get_plane(db)
        except torch.OutOfMemoryError:
            if mode != _lib.FL_KNN_AUTO:
                raise
            # the plane takes half the memory of the fp32 rows again: without room for it, the exact mode
            resolved, passed, wants_plane, ws_bytes, staged_bytes = _knn_plan(lib, dev.index, nq, m, d, k, _lib.FL_KNN_EXACT_SIMT)
    if out is not None:
        out_d, out_i = out
    else:
        out_d = torch.empty((nq, k), dtype=torch.float32, device=dev)
        out_i = torch.empty((nq, k), dtype=torch.int32, device=dev)
    split = None
    if wants_plane and staged_bytes and nq > 0:
        if second_stage is None:
            second_stage = _second_stage_default()
        if second_stage:
            try:
                split = plane.split_ptr(db)
            except torch.OutOfMemoryError:
                pass               # rows the first proof rejects take the exact pass at once
            if split is not None:
                ws_bytes = staged_bytes
    # (the kernels clear the status words themselves)
    status = torch.empty(_lib.FL_STATUS_WORDS, dtype=torch.int32, device=dev) if nq else torch.zeros(_lib.FL_STATUS_WORDS, dtype=torch.int32, device=dev)
    ws = torch.empty(max(ws_bytes, 1), dtype=torch.uint8, device=dev)
    slot = None
    if check_status == "deferred" and wants_plane and nq and not torch.cuda.is_current_stream_capturing():
        slot = _take_status_slot(dev)
    rc = lib.fl_knn_search(q.data_ptr(), nq, q.stride(0) if nq else d, db.data_ptr(), m, db.stride(0), d, k,
                           _DTYPE_CODES[db.dtype], passed, plane.ptr if plane is not None else None, split, row_offset,
                           out_d.data_ptr(), out_i.data_ptr(), ws.data_ptr(), ws_bytes, status.data_ptr(),
                           slot.ptr if slot is not None else None, _stream_ptr(dev))
    if rc != _lib.FL_OK:
        _lib.check(rc)
    if slot is not None:
        _PENDING_STATUS.append(slot)
    info = {"mode": resolved, "status": status, "second_stage": split is not None}
    if check_status and check_status != "deferred" and wants_plane:
        st = status.tolist()
        info["fallback_rows"] = st[_lib.FL_STATUS_FALLBACK]
        info["stage2_rows"] = st[_lib.FL_STATUS_STAGE2]
        _raise_on_status(st)
    return out_d, out_i, info


def flash_knn_dispatch(x: torch.Tensor, c: torch.Tensor, k: int, *, tol: Optional[float] = None,
                       backend: Optional[str] = None, return_distances: bool = True,
                       mode: Optional[str] = None, **kwargs):
    """Exact k nearest rows of ``c`` for every row of ``x`` by squared L2.

    Parameters follow ``flashlib/primitives/knn/impl.py:199-247``: ``x`` is ``(B, N, D)`` or
    ``(N, D)``, ``c`` has the same rank and dtype, ``backend`` may be ``None`` or one of the
    reference's names (validated, then ignored: there is one implementation).  bf16 / fp16
    inputs are read as stored (no fp32 copy); ``tol`` follows the reference's rule
    (``storage_dtype_for``): when it allows 16-bit storage, fp32 inputs are cast to it -- the
    database once, cached -- and the result is the exact kNN of the stored values, as in the
    reference (``knn/impl.py:257-261``).  ``mode`` (``"exact"`` | ``"bf16"`` | ``None`` = auto)
    picks the scoring kernel.

    Returns ``(vals, idxs)`` -- fp32 true squared distances ascending and int32 indices --
    or just ``idxs`` with ``return_distances=False``.
    """
    if backend is not None and backend not in _VALID_BACKENDS:
        raise ValueError(f"backend must be one of {_VALID_BACKENDS} or None, got {backend!r}")
    if x.dim() not in (2, 3) or c.dim() != x.dim():
        raise ValueError("flash_knn expects x and c of the same rank: (N, D)/(M, D) or (B, N, D)/(B, M, D)")
    if x.dtype != c.dtype:
        raise AssertionError("x and c must share a dtype")
    if not (x.is_cuda and c.is_cuda):
        raise RuntimeError("flashlib_b200.flash_knn needs CUDA tensors (no CPU fallback)")
    squeeze = x.dim() == 2
    if squeeze:
        x = x.unsqueeze(0)
        c = c.unsqueeze(0)
    B, N, D = x.shape
    Bc, M, Dc = c.shape
    if Bc != B or Dc != D:
        raise AssertionError("x and c must agree on batch and feature dimensions")
    if not (1 <= int(k) <= M):
        raise AssertionError(f"k must be in [1, M={M}] (got {k})")
    k = int(k)
    m = _mode_from(mode)
    vals = torch.empty((B, N, k), dtype=torch.float32, device=x.device)
    idxs = torch.empty((B, N, k), dtype=torch.int32, device=x.device)
    target = storage_dtype_for(tol)
    lib = _lib.load()
    if B == 1:
        with _OnDevice(x.device):
            qb, cb = x[0], c[0]
            if target is not None and qb.dtype != target:
                qb, cb = qb.to(target), _cast_rows_cached(cb, target)
            knn_f32(_as_rows(qb), _as_rows(cb), k, mode=m, check_status="deferred", out=(vals[0], idxs[0]))
        if not return_distances:
            return idxs[0] if squeeze else idxs
        return (vals[0], idxs[0]) if squeeze else (vals, idxs)
    batched = (B > 1 and N > 0 and target is None and x.dtype == torch.float32 and m != _lib.FL_KNN_BF16_RERANK
               and lib.fl_knn_batch_route(B, N, M, D, k)
               and x.stride(2) == 1 and c.stride(2) == 1 and x.stride(1) >= D and c.stride(1) >= D)
    if batched:
        # many small problems: one launch sequence for the whole batch
        _lib.require_device()
        with torch.cuda.device(x.device):
            ws_bytes = lib.fl_knn_batch_workspace_bytes(B, N, M, D, k)
            ws = torch.empty(ws_bytes, dtype=torch.uint8, device=x.device)
            _lib.check(lib.fl_knn_batch_f32(x.data_ptr(), B, N, x.stride(1), x.stride(0), c.data_ptr(), M, c.stride(1),
                                            c.stride(0), D, k, vals.data_ptr(), idxs.data_ptr(), ws.data_ptr(), ws_bytes,
                                            _stream_ptr(x.device)))
        if not return_distances:
            return idxs
        return vals, idxs
    with torch.cuda.device(x.device):
        for b in range(B):
            qb, cb = x[b], c[b]
            if target is not None and qb.dtype != target:
                qb, cb = qb.to(target), _cast_rows_cached(cb, target)
            qb, cb = _as_rows(qb), _as_rows(cb)
            knn_f32(qb, cb, k, mode=m, check_status="deferred", out=(vals[b], idxs[b]))
    if not return_distances:
        return idxs
    return vals, idxs


flash_knn = flash_knn_dispatch
flash_knn_triton = flash_knn_dispatch  # name kept for callers of the reference's Triton entry


def triton_knn_gather_sqdist(x: torch.Tensor, c: torch.Tensor, idx: torch.Tensor,
                             out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``out[b,n,j] = sum_d (x[b,n,d] - c[b,idx[b,n,j],d])^2`` in fp32.

    Same contract as ``flashlib/kernels/distance/triton/knn_gather_l2sq.py:173-229``
    (3-D inputs, int32 or int64 indices).
    """
    assert x.is_cuda and c.is_cuda and idx.is_cuda
    assert x.dim() == 3 and c.dim() == 3 and idx.dim() == 3
    B, N, D = x.shape
    Bc, M, Dc = c.shape
    Bi, Ni, K = idx.shape
    assert B == Bc == Bi and N == Ni and D == Dc
    assert idx.dtype in (torch.int32, torch.int64)
    lib = _lib.load()
    _lib.require_device()
    if out is None:
        out = torch.empty((B, N, K), dtype=torch.float32, device=x.device)
    else:
        assert out.shape == (B, N, K) and out.dtype == torch.float32 and out.is_contiguous()
    with torch.cuda.device(x.device):
        for b in range(B):
            xb = _as_f32_rows(x[b])
            cb = _as_f32_rows(c[b])
            ib = idx[b].contiguous()
            _lib.check(lib.fl_gather_l2sq_f32(xb.data_ptr(), N, xb.stride(0), cb.data_ptr(), M, cb.stride(0), D,
                                              ib.data_ptr(), 1 if ib.dtype == torch.int64 else 0, K,
                                              out[b].data_ptr(), _stream_ptr(x.device)))
    return out


def row_sqnorm(x: torch.Tensor) -> torch.Tensor:
    """fp32 ``||row||^2`` of a 2-D CUDA tensor (``knn/triton/_row_norm.py:59-93``)."""
    lib = _lib.load()
    _lib.require_device()
    xb = _as_f32_rows(x)
    out = torch.empty(xb.shape[0], dtype=torch.float32, device=x.device)
    with torch.cuda.device(x.device):
        _lib.check(lib.fl_rownorm_f32(xb.data_ptr(), xb.shape[0], xb.shape[1], xb.stride(0), out.data_ptr(),
                                      _stream_ptr(x.device)))
    return out


def topk_merge(cand_dist: torch.Tensor, cand_idx: torch.Tensor, k: int):
    """k smallest ``(dist, idx)`` per row of ``(nq, ncand)`` candidates (idx < 0 ignored)."""
    lib = _lib.load()
    _lib.require_device()
    cand_dist = cand_dist.contiguous().float()
    cand_idx = cand_idx.contiguous().to(torch.int32)
    nq, ncand = cand_dist.shape
    out_d = torch.empty((nq, k), dtype=torch.float32, device=cand_dist.device)
    out_i = torch.empty((nq, k), dtype=torch.int32, device=cand_dist.device)
    with torch.cuda.device(cand_dist.device):
        _lib.check(lib.fl_topk_merge_f32(cand_dist.data_ptr(), cand_idx.data_ptr(), nq, ncand, k,
                                         out_d.data_ptr(), out_i.data_ptr(), _stream_ptr(cand_dist.device)))
    return out_d, out_i
