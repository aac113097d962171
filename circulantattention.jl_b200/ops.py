"""Thin tensor-level wrappers over the C ABI: shape bookkeeping, output
allocation (the caller owns every buffer, as CUDA.jl's pool does on the Julia
side) and the ctypes calls.  No arithmetic happens here.  The public API takes the
native route of csrc/host.cpp; the attention wrappers here serve callers that drive
the stages themselves (the band split, the benchmark)."""
from __future__ import annotations

import math
from dataclasses import dataclass

import torch

from . import _lib, jl
from ._lib import CA_BF16, CA_C64, CA_F32, ca_desc, check, host, lib, ptr  # noqa: F401  (re-exported: parallel.py uses ops.lib / ops.check)


@dataclass(frozen=True)
class Meta:
    """What a windowed kernel needs to know about a (spatial..., c, units) tensor."""
    spatial: tuple
    channels: int
    units: int
    ws: int
    cplx: bool
    bf16: bool = False      # bfloat16 storage (fused attention only)

    @property
    def ndim(self):
        return len(self.spatial)

    @property
    def H(self):
        return self.spatial[0]

    @property
    def W(self):
        return self.spatial[1] if len(self.spatial) == 2 else 1

    @property
    def Np(self):
        return self.H * self.W

    @property
    def K(self):
        return self.ws ** self.ndim

    def desc(self, similarity=0, normalizer=0, scale=1.0, Wk=0, wk_off=0, units=None, W=None):
        return ca_desc(self.H, self.W if W is None else W, self.ndim, self.channels,
                       self.units if units is None else units, self.ws,
                       CA_C64 if self.cplx else (CA_BF16 if self.bf16 else CA_F32), similarity, normalizer, Wk, wk_off,
                       float(scale))


def meta_of(x: torch.Tensor, ws: int) -> Meta:
    if x.ndim not in (3, 4):
        raise AssertionError(f"expected a (spatial..., channels, batch) array with 1 or 2 spatial dims, got {tuple(x.shape)}")
    return Meta(tuple(x.shape[:-2]), x.shape[-2], x.shape[-1], int(ws), x.is_complex(), x.dtype == torch.bfloat16)


_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def _stream():
    """Handle (cudaStream_t as an integer) of torch's current stream on the current device."""
    if _raw_stream is not None:
        return _raw_stream(torch.cuda.current_device())
    return torch.cuda.current_stream().cuda_stream


_NVTX = [False]


def enable_nvtx(flag: bool = True) -> bool:
    """NVTX ranges ("circatt.fwd", "circatt.bwd", "circatt.halo") around the library's calls, for timeline
    profilers; off by default (a range costs two host calls).  Returns the previous setting."""
    old, _NVTX[0] = _NVTX[0], bool(flag)
    host.enable_nvtx(bool(flag))
    return old


class _on_device:
    """`with _on_device(t.device)`: makes that device current for the C ABI calls inside, without the cost of
    a device switch when it already is (the common case).  With a `name` and NVTX enabled the block is also
    an NVTX range."""
    __slots__ = ("index", "prev", "name")

    def __init__(self, device, name=None):
        self.index = device.index if device.index is not None else torch.cuda.current_device()
        self.prev = None
        self.name = name if (name and _NVTX[0]) else None

    def __enter__(self):
        cur = torch.cuda.current_device()
        if cur != self.index:
            self.prev = cur
            torch.cuda.set_device(self.index)
        if self.name:
            torch.cuda.nvtx.range_push(self.name)

    def __exit__(self, *exc):
        if self.name:
            torch.cuda.nvtx.range_pop()
        if self.prev is not None:
            torch.cuda.set_device(self.prev)
        return False


def require_cuda(*ts):
    for t in ts:
        if t is not None and not t.is_cuda:
            raise RuntimeError("CirculantAttention is only CUDA compatible (no CPU path): got a tensor on " + str(t.device))


def _dense_ok(t, cplx=None):
    want = (torch.float32, torch.complex64, torch.bfloat16)
    if t.dtype not in want:
        raise TypeError(f"only Float32, ComplexF32 and (fused attention) BFloat16 are supported, got {t.dtype}")
    return jl.colmajor(t)


def structure(spatial, ws, batch, device):
    """rowPtr (Np+1, batch...) and colVal (Np*K, batch...) Int32, 1-based."""
    spatial = tuple(spatial)
    H, W = spatial[0], (spatial[1] if len(spatial) == 2 else 1)
    Np, K = H * W, ws ** len(spatial)
    nb = int(math.prod(batch)) if batch else 1
    rowptr = jl.empty((Np + 1,) + tuple(batch), torch.int32, device)
    colval = jl.empty((Np * K,) + tuple(batch), torch.int32, device)
    with _on_device(rowptr.device):
        check(lib.ca_structure(H, W, len(spatial), ws, nb, ptr(rowptr), ptr(colval), _stream()))
    return rowptr, colval


# ------------------------------------------------------------------ operators on values (native: csrc/host.cpp)
def similarity(kind, x, y, ws, scale=1.0):
    """Scaled scores (Np*K, units) of head-split (spatial..., c, units) tensors."""
    return host.similarity_raw(kind, x, y, ws, scale)


def similarity_bwd(kind, x, y, ws, dS, scale=1.0):
    return host.similarity_bwd_raw(kind, x, y, ws, dS, scale)


def row_normalize(nz, spatial, ws, normalizer, out=None, want_stats=False):
    p, stats = host.normalize_raw(nz, list(spatial), ws, normalizer, out, want_stats)
    return (p, stats) if want_stats else p


def row_normalize_bwd(p, dp, spatial, ws, normalizer):
    return host.normalize_bwd_raw(p, dp, list(spatial), ws, normalizer)


def apply(nz, v, ws, transpose=False, out=None):
    """A (x) v or A^T (x) v.  nz: (Np*K, ua); v: (spatial..., c, uv); ua, uv broadcast."""
    return host.apply_raw(nz, v, ws, bool(transpose), 1, out)


# Transient scratch per (device, stream, purpose): grown on demand and reused by later calls on the
# same stream, which is safe because work on one stream is ordered.  Buffers that must outlive the
# call (the forward workspace kept for the backward) are never taken from here.
_SCRATCH = {}


def _scratch(purpose, nbytes, device):
    if not nbytes:
        return None
    key = (device.index, _stream(), purpose)
    buf = _SCRATCH.get(key)
    if buf is None or buf.numel() < nbytes:
        buf = torch.empty(nbytes, dtype=torch.uint8, device=device)
        _SCRATCH[key] = buf
    return buf


def release_scratch():
    """Drops the cached transient workspaces (they are re-created on demand)."""
    _SCRATCH.clear()


# ------------------------------------------------------------------ device-side failure reporting
def _status_word(device):
    """The int32 on `device` in which kernels flag a wait that ran out; registered with the library for the
    calling host thread."""
    return host.status_word(torch.cuda.current_device() if device.index is None else device.index)


def check_status(device=None):
    """Synchronising check: raises if a kernel of this library gave up a bounded device-side wait since the
    last check on `device` (its tile then holds NaN).  Call it where the program synchronises anyway."""
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    index = torch.cuda.current_device() if device.index is None else device.index
    if not host.has_status_word(index):
        return
    w = host.status_word(index)
    flag = int(w.item())
    if flag:
        w.zero_()
        raise _lib.CircAttError("a circatt_b200 kernel gave up a bounded wait for a shared-memory stage copy; "
                                "the outputs of that call hold NaN")


def attention_fwd(kind, normalizer, q, k, v, ws, want_nz, scale=None, band=None, keep_workspace=False):
    """Fused forward on (spatial..., c, units) tensors.  Returns (y, nz | None, stats), plus the workspace
    tensor when `keep_workspace` (hand it to attention_bwd as `fwd_workspace`).
    `band=(Wk, wk_off)` selects band mode: k, v then have Wk columns."""
    require_cuda(q, k, v)
    q, k, v = _dense_ok(q), _dense_ok(k), _dense_ok(v)
    m = meta_of(q, ws)
    scale = 1.0 / math.sqrt(m.channels) if scale is None else scale
    Wk, wk_off = band if band else (0, 0)
    d = m.desc(similarity=kind, normalizer=normalizer, scale=scale, Wk=Wk, wk_off=wk_off)
    y = jl.empty(q.shape, q.dtype, q.device)
    nz = jl.empty((m.Np * m.K, m.units), torch.float32, q.device) if want_nz else None
    stats = jl.empty((m.Np, m.units), torch.float32, q.device)
    nbytes = lib.ca_attention_fwd_workspace(d, int(want_nz))
    with _on_device(q.device, "circatt.fwd"):
        _status_word(q.device)
        if keep_workspace:
            wsb = torch.empty(nbytes, dtype=torch.uint8, device=q.device) if nbytes else None
        else:
            wsb = _scratch("fwd", nbytes, q.device)
        check(lib.ca_attention_fwd(d, ptr(q), ptr(k), ptr(v), ptr(y), ptr(nz), ptr(stats), ptr(wsb), _stream()))
    return (y, nz, stats, wsb) if keep_workspace else (y, nz, stats)


def attention_bwd(kind, normalizer, q, k, v, y, dy, stats, ws, nz=None, dA=None, scale=None, fwd_workspace=None):
    """Fused backward.  Returns (dq, dk, dv).  `fwd_workspace`: the workspace kept from the matching
    attention_fwd(keep_workspace=True) call, untouched since (spares packing k and v again)."""
    q, k, v, y, dy = (_dense_ok(t) for t in (q, k, v, y, dy))
    m = meta_of(q, ws)
    scale = 1.0 / math.sqrt(m.channels) if scale is None else scale
    d = m.desc(similarity=kind, normalizer=normalizer, scale=scale)
    dq, dk, dv = (jl.empty(q.shape, q.dtype, q.device) for _ in range(3))
    if dA is not None:
        dA = jl.colmajor(dA)
    with _on_device(q.device, "circatt.bwd"):
        _status_word(q.device)
        wsb = _scratch("bwd", lib.ca_attention_bwd_workspace(d, int(dA is not None)), q.device)
        check(lib.ca_attention_bwd(d, ptr(q), ptr(k), ptr(v), ptr(y), ptr(dy), ptr(stats), ptr(nz), ptr(dA),
                                   ptr(dq), ptr(dk), ptr(dv), ptr(wsb), ptr(fwd_workspace), _stream()))
    return dq, dk, dv


def copy_chunks(jobs):
    """Several strided device copies in one launch (ca_copy_chunks).  `jobs`: tuples
    (src_ptr, dst_ptr, chunk_bytes, nchunks, src_stride_bytes, dst_stride_bytes) with integer addresses;
    longer lists are split into launches of CA_MAX_CHUNK_JOBS."""
    for i in range(0, len(jobs), _lib.CA_MAX_CHUNK_JOBS):
        part = jobs[i:i + _lib.CA_MAX_CHUNK_JOBS]
        arr = (_lib.ca_chunk_job * len(part))(*[_lib.ca_chunk_job(*j) for j in part])
        check(lib.ca_copy_chunks(arr, len(part), _stream()))


def entmax_scratch_limit(nbytes: int = -1) -> int:
    """Largest A-sized scratch (bytes) the flash-mode entmax forward may use before it switches to the
    scratch-free sweeps; sets it when `nbytes` >= 0.  Returns the previous limit."""
    return int(lib.ca_entmax_scratch_limit(int(nbytes)))


# ------------------------------------------------------------------ algebra (native: csrc/host.cpp)
def axpby(alpha, x, beta=0.0, y=None):
    return host.axpby_raw(float(alpha), x, float(beta), y)


def scale_batch(c, nz):
    """nz (inner, a...) times c (c...) with Julia-style extent-1 broadcasting."""
    return host.scale_batch_raw(c, nz)


def dot_batch(x, y=None):
    """per-slice sum_n x*y (y None: sum of x); x, y: (inner, b...) broadcasting -> (b...)"""
    return host.dot_batch(x, y)


def sum_batch(nz, sum1, sum2):
    return host.sum_batch(nz, bool(sum1), bool(sum2))


def sum_rows(nz, spatial, ws):
    return host.sum_axis(nz, list(spatial), ws, True)


def sum_cols(nz, spatial, ws):
    return host.sum_axis(nz, list(spatial), ws, False)


# ------------------------------------------------------------------ backward stages (band split)
def _stage_ws(d, device):
    n = lib.ca_attention_bwd_stage_workspace(d)
    return torch.empty(max(n, 16), dtype=torch.uint8, device=device) if n else None


def attention_bwd_pre(kind, normalizer, q, k, v, y, dy, stats, ws, scale=None):
    """D of ca_attention_bwd_pre for band-local tensors (no A cotangent)."""
    q, k, v, y, dy = (_dense_ok(t) for t in (q, k, v, y, dy))
    m = meta_of(q, ws)
    scale = 1.0 / math.sqrt(m.channels) if scale is None else scale
    d = m.desc(similarity=kind, normalizer=normalizer, scale=scale)
    D = jl.empty((m.Np, m.units), torch.float32, q.device)
    with _on_device(q.device):
        check(lib.ca_attention_bwd_pre(d, ptr(q), ptr(k), ptr(v), ptr(y), ptr(dy), ptr(stats), None, None, ptr(D),
                                       _stream()))
    return D


def attention_bwd_dq(kind, normalizer, q, k, v, dy, stats, D, ws, scale=None, band=None):
    """dq stage; in band mode k, v carry Wk = W + 2p columns."""
    q, k, v, dy = (_dense_ok(t) for t in (q, k, v, dy))
    m = meta_of(q, ws)
    scale = 1.0 / math.sqrt(m.channels) if scale is None else scale
    Wk, wk_off = band if band else (0, 0)
    d = m.desc(similarity=kind, normalizer=normalizer, scale=scale, Wk=Wk, wk_off=wk_off)
    dq = jl.empty(q.shape, q.dtype, q.device)
    wsb = _stage_ws(d, q.device)
    with _on_device(q.device):
        check(lib.ca_attention_bwd_dq(d, ptr(q), ptr(k), ptr(v), ptr(dy), ptr(stats), ptr(D), None, ptr(dq),
                                      ptr(wsb), _stream()))
    return dq


def attention_bwd_dkdv(kind, normalizer, q, k, v, dy, stats, D, ws, scale=None, band=None):
    """dk/dv stage; in band mode q, dy, stats, D carry Wk = W + 2p columns and k, v are band-local."""
    q, k, v, dy = (_dense_ok(t) for t in (q, k, v, dy))
    m = meta_of(k, ws)
    scale = 1.0 / math.sqrt(m.channels) if scale is None else scale
    Wk, wk_off = band if band else (0, 0)
    d = m.desc(similarity=kind, normalizer=normalizer, scale=scale, Wk=Wk, wk_off=wk_off)
    dk, dv = jl.empty(k.shape, k.dtype, k.device), jl.empty(k.shape, k.dtype, k.device)
    wsb = _stage_ws(d, k.device)
    with _on_device(k.device):
        check(lib.ca_attention_bwd_dkdv(d, ptr(q), ptr(k), ptr(v), ptr(dy), ptr(stats), ptr(D), None, ptr(dk),
                                        ptr(dv), ptr(wsb), _stream()))
    return dk, dv
