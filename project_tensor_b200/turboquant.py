"""TurboQuant quantizers with the public surface of Project-Tensor's ``tensor_gpu_v2/_quant.py``
and all array arithmetic in hand-written sm_100a kernels (libtq_sm100.so, called through ctypes).

Same names, constructor keywords, method names, encoding field names and ``ValueError`` texts as
the reference (``TurboQuantMSE`` _quant.py:172-254, ``TurboQuantProd`` :257-358, encodings
:156-169, helpers :361-374).  What differs, on purpose:

* Inputs may be NumPy arrays, anything exposing ``__cuda_array_interface__`` (CuPy arrays, torch
  CUDA tensors, ...) or a ``Tensor``-like wrapper whose ``.data`` is one of those.  Every input is
  computed on the GPU; NumPy callers get NumPy results back, device callers get device arrays.
  There is no CPU path: without a CUDA device (or without the built library) calls raise.
* Arithmetic is float32, like the reference's documented use; other float dtypes are cast.
* Encodings keep bit-packed device buffers (``d*bits/8`` bytes of codes and ``d/8`` bytes of QJL
  signs per vector).  ``encoding.indices`` / ``encoding.qjl`` unpack on first access into the
  reference's ``uint8 (N, d)`` / ``int8 (N, d)`` arrays.
* ``bits`` above 8 for the MSE stage and ``dimension`` above 1024 are rejected.
* ``TurboQuantProd.attention_scores`` (plural) is an addition: many queries against shared keys
  in one pass, optionally with a fused per-query top-k.  The reference's users obtain the same
  matrix by calling ``attention_score`` once per query.
"""
from __future__ import annotations

import ctypes
import math
import sys
from dataclasses import dataclass
from typing import Any, Dict, Optional, Tuple

import numpy as np

from . import _native
from .codebook import (_build_lloyd_max_codebook, _random_orthogonal_matrix,
                       _random_projection_matrix)

_MAX_BITS = 8
_MAX_DIM = 1024


# ------------------------------------------------------------------------------------------------
# small host helpers
# ------------------------------------------------------------------------------------------------
class Tensor:
    """Minimal stand-in for the reference's ``Tensor``: a holder whose ``.data`` is the array.
    The quantizers only ever read ``.data`` (_quant.py:27-34); no autograd lives here."""

    def __init__(self, data, requires_grad: bool = False):
        self.data = data
        self.requires_grad = bool(requires_grad)

    @property
    def shape(self):
        return self.data.shape


def _torch():
    import torch  # imported lazily: constructing a quantizer needs NumPy only
    return torch


def _is_device_array(obj: Any) -> bool:
    return hasattr(obj, "__cuda_array_interface__")


def _to_array(data: Any):
    """Unwrap a ``Tensor``-like object; leave arrays alone (_quant.py:31-34)."""
    torch = _torch_if_loaded()
    if torch is not None and isinstance(data, torch.Tensor):   # before the attribute test, which builds a dict for a tensor
        return data
    if isinstance(data, np.ndarray) or _is_device_array(data):
        return data
    if isinstance(data, Tensor) or (hasattr(data, "data") and hasattr(data, "requires_grad")):
        return data.data
    return np.asarray(data)


def _torch_if_loaded():
    return sys.modules.get("torch")


def _ensure_last_dim(array, dim: int) -> None:
    if array.ndim == 0 or array.shape[-1] != dim:
        raise ValueError(
            f"expected input with trailing dimension {dim}, got shape {tuple(array.shape)}"
        )


def _quant_index_dtype(bits: int):
    if bits <= 8:
        return np.uint8
    if bits <= 16:
        return np.uint16
    return np.int32


class _Staged:
    """An input brought to the GPU as a contiguous float32 torch tensor of ``n`` rows (its last dimension is d; the
    others are left as the caller had them), remembering what kind of array the caller used so that results can be
    handed back in the same kind."""

    __slots__ = ("tensor", "prefix", "kind", "device", "n")

    def __init__(self, tensor, prefix, kind, device):
        self.tensor, self.prefix, self.kind, self.device = tensor, prefix, kind, device
        self.n = math.prod(prefix)


def _require_cuda():
    torch = _torch()
    if not torch.cuda.is_available():
        raise _native.TurboQuantNativeError(
            "TurboQuant needs a CUDA device (B200, sm_100a); there is no CPU fallback")
    return torch


def _stage(data: Any, dim: int, device=None, halves: bool = False) -> _Staged:
    """``halves``: the caller's kernel reads bf16 and fp16 vectors itself, so CUDA tensors of those types stay as they are
    (see ``_dtype_code``)."""
    torch = _torch_if_loaded()
    if torch is not None and type(data) is torch.Tensor and data.is_cuda:
        # the common device caller: looked at once, nothing converted, no view made (a few microseconds of every call)
        shape = data.shape
        if not shape or shape[-1] != dim:
            _ensure_last_dim(data, dim)
        dtype = data.dtype
        if dtype is not torch.float32 and not (halves and (dtype is torch.bfloat16 or dtype is torch.float16)):
            data = data.to(torch.float32)
        return _Staged(data if data.is_contiguous() else data.contiguous(), tuple(shape[:-1]), "torch", data.device)
    array = _to_array(data)
    _ensure_last_dim(array, dim)
    prefix = tuple(array.shape[:-1])
    torch = _require_cuda()
    if isinstance(array, np.ndarray):
        dev = torch.device("cuda", torch.cuda.current_device()) if device is None else device
        host = torch.from_numpy(np.ascontiguousarray(array, dtype=np.float32))
        # The copy is enqueued and not waited for.  Pageable memory has been read when the call returns (the driver
        # stages it); a page-locked source is the caller's to leave alone until the stream has passed the copy.
        return _Staged(host.to(dev, non_blocking=True), prefix, "numpy", dev)
    if isinstance(array, torch.Tensor):
        if array.is_cuda:
            return _Staged(array.to(torch.float32).contiguous(), prefix, "torch", array.device)
        dev = torch.device("cuda", torch.cuda.current_device()) if device is None else device
        return _Staged(array.to(torch.float32).contiguous().to(dev), prefix, "torch_cpu", dev)
    # CuPy or any other __cuda_array_interface__ producer: zero-copy view
    t = torch.as_tensor(array, device="cuda")
    kind = "cupy" if type(array).__module__.split(".")[0] == "cupy" else "torch"
    return _Staged(t.to(torch.float32).contiguous(), prefix, kind, t.device)


def _dtype_code(tensor) -> int:
    torch = _torch()
    return {torch.float32: _native.TQ_F32, torch.bfloat16: _native.TQ_BF16, torch.float16: _native.TQ_F16}[tensor.dtype]


_MAPPED_BYTES = 1 << 16


def _stage_query(data: Any, dim: int, device) -> _Staged:
    """Queries of a call that waits for its results before it returns.  A few NumPy queries go into a page-locked block
    that the kernels read where it lies (one copy on the host instead of a copy through the driver, 7 us less); the
    block is free again when the call is over."""
    if isinstance(data, np.ndarray) and 0 < data.size * 4 <= _MAPPED_BYTES and device.type == "cuda":
        _ensure_last_dim(data, dim)
        block = _torch().empty(data.shape, dtype=_torch().float32, device="cpu", pin_memory=True)
        block.numpy()[...] = data
        return _Staged(block, tuple(data.shape[:-1]), "numpy", device)
    staged = _stage(data, dim, device=device)
    if staged.tensor.device != device:
        staged.tensor = staged.tensor.to(device)
    return staged


def _deliver(tensor, kind: str, plans: "Optional[_PlanSet]" = None):
    """Hand a device tensor back in the caller's kind of array.  A result that goes to host memory synchronises
    anyway; with ``plans`` the status word of the kernels is read at that point, so that the output of a kernel
    that gave up on a bounded wait is never handed out as if it were complete."""
    if kind == "torch":
        return tensor
    if kind == "numpy":
        return _to_host(tensor, plans).numpy()
    if kind == "torch_cpu":
        return _to_host(tensor, plans)
    if kind == "cupy":
        try:
            import cupy
            return cupy.asarray(tensor)
        except ImportError:  # CuPy-like producer without CuPy importable: give the torch view
            return tensor
    return tensor


_PINNED_FROM_BYTES = 1 << 20


def _to_host(tensor, plans: "Optional[_PlanSet]" = None):
    """Device tensor -> CPU tensor, the status of ``plans`` checked behind the copy: one synchronisation in all.
    Every result comes down into page-locked memory from torch's caching host allocator.  From a megabyte on the caller
    gets that block itself (it goes back to the cache when the array that wraps it dies): a copy into pageable memory
    runs at a few GB/s, so that the 128 MiB score matrix of 32 queries x 1,048,576 keys took 62 ms to hand back, against
    3 ms at the rate of the link.  Smaller results are copied out of the block on the host, so that arrays a caller
    collects by the thousand do not pin memory; a device-to-host copy straight into pageable memory costs 14 us."""
    torch = _torch()
    if tensor.device.type != "cuda":
        return tensor
    host = torch.empty(tensor.shape, dtype=tensor.dtype, device="cpu", pin_memory=True)
    host.copy_(tensor, non_blocking=True)
    if plans is not None:
        plans.check_status(tensor.device)      # waits for the stream
    else:
        torch.cuda.current_stream(tensor.device).synchronize()
    return host if host.numel() * host.element_size() >= _PINNED_FROM_BYTES else host.clone()


def _ptr(t) -> int:
    return 0 if t is None else t.data_ptr()


def _device_index(device) -> int:
    index = device.index
    return _torch().cuda.current_device() if index is None else index


def _stream_ptr(device) -> int:
    """The current stream's handle (torch.cuda.current_stream(device).cuda_stream builds an object for it: 2 us)."""
    return _torch()._C._cuda_getCurrentRawStream(_device_index(device))


# ------------------------------------------------------------------------------------------------
# plans: one set of device constants per (quantizer, GPU)
# ------------------------------------------------------------------------------------------------
class _PlanSet:
    """Lazily created tq_plan handles of one quantizer, one per CUDA device index."""

    def __init__(self, dimension, bits_mse, rotation, codebook, projection):
        self.dimension, self.bits_mse = dimension, bits_mse
        self._rotation = np.ascontiguousarray(rotation, dtype=np.float32)
        self._codebook = np.ascontiguousarray(codebook, dtype=np.float32)
        self._projection = None if projection is None else np.ascontiguousarray(projection, dtype=np.float32)
        self._plans: Dict[int, int] = {}
        self._row_bytes = (4 * ((dimension * bits_mse + 31) // 32), 4 * ((dimension + 31) // 32))
        self._path = _native.TQ_PATH_AUTO

    def handle(self, device) -> int:
        idx = _device_index(device)
        h = self._plans.get(idx)
        if h is None:
            lib = _native.load()
            out = ctypes.c_void_p()
            proj = None if self._projection is None else self._projection.ctypes.data
            _native.check(lib.tq_plan_create(self.dimension, self.bits_mse, self._rotation.ctypes.data,
                                             self._codebook.ctypes.data, proj, idx, ctypes.byref(out)))
            h = out.value
            if self._path != _native.TQ_PATH_AUTO:
                _native.check(lib.tq_plan_set_path(h, self._path))
            self._plans[idx] = h
        return h

    def check_status(self, device) -> None:
        """Raise if a tensor-core kernel of this quantizer gave up on a bounded wait on ``device`` since the last
        check.  Synchronises the current stream of that device in any case: callers rely on it to have waited for the copies they
        enqueued, also for an encoding whose quantizer has not been used on the device yet (one read from a file)."""
        h = self._plans.get(_device_index(device))
        if h is None:
            _torch().cuda.current_stream(device).synchronize()
            return
        status = ctypes.c_int64(0)
        _native.check(_native.load().tq_plan_status(h, _stream_ptr(device), ctypes.byref(status)))
        if status.value:
            self.refuse(status.value)

    @staticmethod
    def refuse(status: int) -> None:
        what = {1: "quantize", 2: "scoring", 3: "dequantize"}.get(status, "tensor-core")
        raise _native.TurboQuantNativeError(
            f"a {what} kernel gave up on a bounded wait (status {status}); the results of the calls "
            f"since the last check are incomplete")

    def set_wait_limit(self, cycles: int) -> None:
        """Limit of one bounded wait inside the tensor-core kernels, in GPU cycles, for plans that exist already."""
        for h in self._plans.values():
            _native.check(_native.load().tq_plan_set_wait_limit(h, int(cycles)))

    def set_path(self, path: int) -> None:
        self._path = path
        lib = _native.load()
        for h in self._plans.values():
            _native.check(lib.tq_plan_set_path(h, path))

    def row_bytes(self) -> Tuple[int, int]:
        """(code row bytes, sign row bytes); same formula as the library, usable without a GPU."""
        return self._row_bytes

    def __del__(self):
        try:
            lib = _native.load()
            for h in self._plans.values():
                lib.tq_plan_destroy(h)
        except Exception:
            pass


# ------------------------------------------------------------------------------------------------
# encodings
# ------------------------------------------------------------------------------------------------
class _Packed:
    """Device-resident form of an encoding: bit-packed rows plus per-row float32 scalars."""

    __slots__ = ("codes", "signs", "norms", "residual_norms", "n", "kind", "device", "plans")

    def __init__(self, codes, signs, norms, residual_norms, n, kind, device, plans):
        self.codes, self.signs, self.norms, self.residual_norms = codes, signs, norms, residual_norms
        self.n, self.kind, self.device, self.plans = n, kind, device, plans


def _lazy_field(name: str, make):
    slot = "_" + name

    def getter(self):
        value = self.__dict__.get(slot)
        if value is None and self.__dict__.get("_packed") is not None:
            value = make(self.__dict__["_packed"])
            self.__dict__[slot] = value
        return value

    def setter(self, value):
        self.__dict__[slot] = value

    return property(getter, setter)


def _unpack_codes(pk: _Packed):
    torch = _torch()
    out = torch.empty((pk.n, pk.plans.dimension), dtype=torch.uint8, device=pk.device)
    if pk.n:
        _native.check(_native.load().tq_unpack_codes(pk.plans.handle(pk.device), _ptr(pk.codes), pk.n,
                                                     _ptr(out), _stream_ptr(pk.device)))
    return _deliver(out, pk.kind, pk.plans)


def _unpack_signs(pk: _Packed):
    torch = _torch()
    out = torch.empty((pk.n, pk.plans.dimension), dtype=torch.int8, device=pk.device)
    if pk.n:
        _native.check(_native.load().tq_unpack_signs(pk.plans.handle(pk.device), _ptr(pk.signs), pk.n,
                                                     _ptr(out), _stream_ptr(pk.device)))
    return _deliver(out, pk.kind, pk.plans)


@dataclass
class TurboQuantMSEEncoding:
    indices: Any
    norms: Any
    prefix_shape: Tuple[int, ...]


@dataclass
class TurboQuantProdEncoding:
    indices: Any
    qjl: Any
    residual_norms: Any
    norms: Any
    prefix_shape: Tuple[int, ...]


# The dataclass fields above stay what ``dataclasses.fields`` reports; the array-valued ones are
# served by properties so that encodings produced here can keep packed device buffers and only
# materialise the reference-shaped arrays when somebody reads them.
for _cls in (TurboQuantMSEEncoding, TurboQuantProdEncoding):
    _cls.indices = _lazy_field("indices", _unpack_codes)
    _cls.norms = _lazy_field("norms", lambda pk: _deliver(pk.norms, pk.kind, pk.plans))
TurboQuantProdEncoding.qjl = _lazy_field("qjl", _unpack_signs)
TurboQuantProdEncoding.residual_norms = _lazy_field(
    "residual_norms", lambda pk: _deliver(pk.residual_norms, pk.kind, pk.plans))


def _row_shape(rows: int, prefix) -> Tuple[int, ...]:
    """Shape to allocate the results of ``rows`` rows in: ``prefix`` when it holds them as it stands, else flat -- the field
    ``prefix_shape`` can be edited, and ``reshape`` then says what it makes of it (a -1 in it, or no such shape)."""
    prefix = tuple(prefix)
    return prefix if math.prod(prefix) == rows and (len(prefix) < 2 or min(prefix) >= 0) else (rows,)


def _in_shape(result, shape):
    return result if result.shape == shape else result.reshape(shape)


def _encoding_from_packed(cls, pk: _Packed, prefix):
    enc = cls.__new__(cls)
    enc.__dict__["_packed"] = pk
    enc.__dict__["prefix_shape"] = tuple(prefix)
    return enc


def packed_buffers(encoding) -> Dict[str, Any]:
    """The device buffers behind an encoding produced by this package, as torch tensors:
    ``codes`` uint8 (N, code_row_bytes), ``signs`` uint8 (N, sign_row_bytes) or None, ``norms``
    and ``residual_norms`` float32 (N,).  Raises for encodings built by hand from arrays."""
    pk = encoding.__dict__.get("_packed")
    if pk is None:
        raise ValueError("this encoding holds plain arrays, not packed device buffers")
    return {"codes": pk.codes, "signs": pk.signs, "norms": pk.norms, "residual_norms": pk.residual_norms}


def packed_to_host(encoding, out: Optional[Dict[str, Any]] = None, wait: bool = True) -> Dict[str, Any]:
    """Copy the packed buffers of an encoding into page-locked host tensors (same keys as
    ``packed_buffers``).  ``out`` may be the dict returned by an earlier call for an encoding of the
    same shape; its tensors are reused, which avoids allocating (and faulting in) fresh host memory for
    every batch -- a device-to-host copy into new pageable memory runs far below the link rate.  The
    copies are enqueued on the current stream; with ``wait=False`` the caller synchronises."""
    torch = _require_cuda()
    bufs = packed_buffers(encoding)
    host: Dict[str, Any] = {} if out is None else out
    for name, dev_t in bufs.items():
        if dev_t is None:
            host[name] = None
            continue
        dst = host.get(name)
        if dst is None or dst.shape != dev_t.shape or dst.dtype != dev_t.dtype or not dst.is_pinned():
            dst = torch.empty(dev_t.shape, dtype=dev_t.dtype, device="cpu", pin_memory=True)
            host[name] = dst
        dst.copy_(dev_t, non_blocking=True)
    if wait:
        pk = encoding.__dict__["_packed"]
        pk.plans.check_status(pk.device)     # synchronises the stream, and refuses results of a kernel that gave up
    return host


#: a last chunk of so few rows would be quantized by another kernel than the rest
_SHORT_CHUNK_ROWS = 8192


def quantize_to_host(quantizer, keys, chunk_rows: int = 131072, out: Optional[Dict[str, Any]] = None) -> Dict[str, Any]:
    """Quantize host-resident keys and leave the packed encoding in page-locked host tensors, for key sets
    that do not stay on the GPU (``quantizer`` is a TurboQuantMSE or TurboQuantProd, ``keys`` a NumPy
    array of shape (..., d), best page-locked).  The keys go up in chunks of ``chunk_rows`` on one stream
    while the previous chunk is quantized on a second and the chunk before that is copied back on a third,
    so the call takes about as long as the host-to-device copy alone.  Returns the dict described under
    ``packed_buffers`` (``out`` may be the dict of an earlier call of the same size: its tensors are
    reused)."""
    torch = _require_cuda()
    prod = isinstance(quantizer, TurboQuantProd)
    mseq = quantizer.mse if prod else quantizer
    plans = quantizer._plans
    d = quantizer.dimension
    array = _to_array(keys)
    if not isinstance(array, np.ndarray):
        raise TypeError("quantize_to_host expects host (NumPy) keys; use quantize() for device arrays")
    _ensure_last_dim(array, d)
    flat = torch.from_numpy(np.ascontiguousarray(array.reshape(-1, d), dtype=np.float32))
    n = flat.shape[0]
    device = torch.device("cuda", torch.cuda.current_device())
    code_bytes, sign_bytes = plans.row_bytes()
    shapes = {"codes": ((n, code_bytes), torch.uint8), "norms": ((n,), torch.float32)}
    if prod:
        shapes.update({"signs": ((n, sign_bytes), torch.uint8), "residual_norms": ((n,), torch.float32)})
    host: Dict[str, Any] = {} if out is None else out
    for name, (shape, dtype) in shapes.items():
        t = host.get(name)
        if t is None or tuple(t.shape) != shape or t.dtype != dtype or not t.is_pinned():
            host[name] = torch.empty(shape, dtype=dtype, device="cpu", pin_memory=True)
    if not prod:
        host["signs"] = host["residual_norms"] = None
    if n == 0:
        return host
    chunk_rows = max(1, min(int(chunk_rows), n))
    if 0 < n % chunk_rows <= _SHORT_CHUNK_ROWS < chunk_rows:
        chunk_rows = -(-n // -(-n // chunk_rows))    # chunks of one size
    with torch.cuda.device(device):
        s_in, s_run, s_out = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.Stream()
        for s_ in (s_in, s_run, s_out):
            s_.wait_stream(torch.cuda.current_stream())
        bufs = [torch.empty((chunk_rows, d), dtype=torch.float32, device=device) for _ in range(2)]
        ran = [None, None]          # event: the kernels that read bufs[b] have finished
        alive = []                  # chunk results stay allocated until the copies back are done
        for i, start in enumerate(range(0, n, chunk_rows)):
            m = min(chunk_rows, n - start)
            b = i & 1
            with torch.cuda.stream(s_in):
                if ran[b] is not None:
                    s_in.wait_event(ran[b])
                bufs[b][:m].copy_(flat[start:start + m], non_blocking=True)
                up = torch.cuda.Event()
                up.record(s_in)
            with torch.cuda.stream(s_run):
                s_run.wait_event(up)
                pk = mseq._quantize_staged(_Staged(bufs[b][:m], (m,), "torch", device), plans, prod)
                ran[b] = torch.cuda.Event()
                ran[b].record(s_run)
            with torch.cuda.stream(s_out):
                s_out.wait_event(ran[b])
                host["codes"][start:start + m].copy_(pk.codes, non_blocking=True)
                host["norms"][start:start + m].copy_(pk.norms, non_blocking=True)
                if prod:
                    host["signs"][start:start + m].copy_(pk.signs, non_blocking=True)
                    host["residual_norms"][start:start + m].copy_(pk.residual_norms, non_blocking=True)
            alive.append(pk)
        s_out.synchronize()
        torch.cuda.current_stream().wait_stream(s_run)
        plans.check_status(device)     # a chunk whose kernel gave up on a bounded wait must not pass as quantized
    return host


def _as_packed(encoding, plans: _PlanSet, need_signs: bool) -> _Packed:
    """Packed device form of ``encoding``: its own buffers when it came from this quantizer's
    geometry, else packed now from the reference-style array fields."""
    pk = encoding.__dict__.get("_packed")
    if pk is not None and pk.plans.dimension == plans.dimension and pk.plans.bits_mse == plans.bits_mse:
        if pk.plans is not plans:
            pk = _Packed(pk.codes, pk.signs, pk.norms, pk.residual_norms, pk.n, pk.kind, pk.device, plans)
        return pk
    torch = _require_cuda()
    lib = _native.load()
    indices = _to_array(encoding.indices)
    d = plans.dimension
    if isinstance(indices, np.ndarray):
        kind = "numpy"
        device = torch.device("cuda", torch.cuda.current_device())
        to_dev = lambda a, dt: torch.from_numpy(np.ascontiguousarray(a)).to(device).to(dt).contiguous()
    else:
        kind = "torch"
        first = torch.as_tensor(indices, device="cuda") if not isinstance(indices, torch.Tensor) else indices
        device = first.device if first.is_cuda else torch.device("cuda", torch.cuda.current_device())
        kind = "torch" if first.is_cuda else "torch_cpu"
        to_dev = lambda a, dt: (a if isinstance(a, torch.Tensor) else torch.as_tensor(a, device="cuda")).to(device).to(dt).contiguous()
    idx = to_dev(indices, torch.uint8)
    if idx.ndim != 2 or idx.shape[1] != d:
        raise ValueError(f"expected indices of shape (N, {d}), got {tuple(idx.shape)}")
    n = idx.shape[0]
    code_bytes, sign_bytes = plans.row_bytes()
    handle = plans.handle(device)
    codes = torch.empty((n, code_bytes), dtype=torch.uint8, device=device)
    norms = to_dev(_to_array(encoding.norms), torch.float32).reshape(-1)
    signs = rnorms = None
    with torch.cuda.device(device):
        st = _stream_ptr(device)
        if n:
            _native.check(lib.tq_pack_codes(handle, _ptr(idx), n, _ptr(codes), st))
        if need_signs:
            qjl = to_dev(_to_array(encoding.qjl), torch.int8)
            signs = torch.empty((n, sign_bytes), dtype=torch.uint8, device=device)
            rnorms = to_dev(_to_array(encoding.residual_norms), torch.float32).reshape(-1)
            if n:
                _native.check(lib.tq_pack_signs(handle, _ptr(qjl), n, _ptr(signs), st))
    return _Packed(codes, signs, norms, rnorms, n, kind, device, plans)


# ------------------------------------------------------------------------------------------------
# quantizers
# ------------------------------------------------------------------------------------------------
class TurboQuantMSE:
    """TurboQuant variant optimized for MSE reconstruction (GPU kernels behind the reference API)."""

    def __init__(self, dimension: int, bits: int, *, seed: Optional[int] = None, grid_size: int = 16385,
                 max_iter: int = 200, rotation: Optional[np.ndarray] = None,
                 codebook: Optional[np.ndarray] = None):
        if dimension < 2:
            raise ValueError("dimension must be >= 2")
        if bits < 1:
            raise ValueError("bits must be >= 1")
        if bits > _MAX_BITS:
            raise ValueError(f"bits must be <= {_MAX_BITS} on the B200 path")
        if dimension > _MAX_DIM:
            raise ValueError(f"dimension must be <= {_MAX_DIM} on the B200 path")
        self.dimension = int(dimension)
        self.bits = int(bits)
        if rotation is not None:
            self.rotation = np.asarray(rotation, dtype=np.float32)
        else:
            self.rotation = _random_orthogonal_matrix(self.dimension, seed)
        if self.rotation.shape != (self.dimension, self.dimension):
            raise ValueError(
                f"rotation must have shape {(self.dimension, self.dimension)}, got {self.rotation.shape}"
            )
        if codebook is not None:
            self.codebook = np.asarray(codebook, dtype=np.float32)
        else:
            self.codebook = _build_lloyd_max_codebook(
                self.dimension, self.bits, grid_size=grid_size, max_iter=max_iter).astype(np.float32)
        if self.codebook.ndim != 1 or self.codebook.shape[0] != (1 << self.bits):
            raise ValueError("codebook shape does not match bit-width")
        self.boundaries = 0.5 * (self.codebook[:-1] + self.codebook[1:])
        self.index_dtype = _quant_index_dtype(self.bits)
        self._plans = _PlanSet(self.dimension, self.bits, self.rotation, self.codebook, None)

    # The tensor-core kernels are used when they exist for (dimension, bits); tests and
    # benchmarks can pin either arithmetic.
    def set_kernel_path(self, path: str) -> None:
        """'auto' | 'exact' | 'tensor' (see TQ_PATH_* in include/tq_b200.h)."""
        self._plans.set_path({"auto": _native.TQ_PATH_AUTO, "exact": _native.TQ_PATH_EXACT,
                              "tensor": _native.TQ_PATH_TENSOR}[path])

    def _quantize_staged(self, staged: _Staged, plans: _PlanSet, prod: bool, out: Optional[Dict[str, Any]] = None) -> _Packed:
        """``out``: contiguous device tensors {codes, norms[, signs, residual_norms]} of n rows to write into
        (e.g. slices of a preallocated index) instead of fresh ones."""
        torch = _torch()
        lib = _native.load()
        x, device, n = staged.tensor, staged.device, staged.n
        code_bytes, sign_bytes = plans.row_bytes()
        handle = plans.handle(device)
        if out:
            codes, norms = out["codes"], out["norms"]
        else:
            codes, norms = x.new_empty((n, code_bytes), dtype=torch.uint8), x.new_empty((n,))
        scratch_bytes = max(lib.tq_quantize_scratch_bytes(handle, n), 16)
        scratch = x.new_empty((scratch_bytes,), dtype=torch.uint8)
        st = _stream_ptr(device)
        if prod:
            if out:
                signs, rnorms = out["signs"], out["residual_norms"]
            else:
                signs, rnorms = x.new_empty((n, sign_bytes), dtype=torch.uint8), x.new_empty((n,))
            _native.check(lib.tq_prod_quantize(handle, x.data_ptr(), n, codes.data_ptr(), signs.data_ptr(), rnorms.data_ptr(),
                                               norms.data_ptr(), scratch.data_ptr(), scratch_bytes, st))
        else:
            signs = rnorms = None
            _native.check(lib.tq_mse_quantize(handle, x.data_ptr(), n, codes.data_ptr(), norms.data_ptr(),
                                              scratch.data_ptr(), scratch_bytes, st))
        return _Packed(codes, signs, norms, rnorms, n, staged.kind, device, plans)

    def quantize(self, vectors: Any) -> TurboQuantMSEEncoding:
        staged = _stage(vectors, self.dimension)
        pk = self._quantize_staged(staged, self._plans, prod=False)
        return _encoding_from_packed(TurboQuantMSEEncoding, pk, staged.prefix)

    def dequantize(self, encoding: TurboQuantMSEEncoding):
        pk = _as_packed(encoding, self._plans, need_signs=False)
        out = pk.norms.new_empty(_row_shape(pk.n, encoding.prefix_shape) + (self.dimension,))
        _native.check(_native.load().tq_mse_dequantize(self._plans.handle(pk.device), pk.codes.data_ptr(),
                                                       pk.norms.data_ptr(), pk.n, out.data_ptr(), _stream_ptr(pk.device)))
        return _in_shape(_deliver(out, pk.kind, pk.plans), tuple(encoding.prefix_shape) + (self.dimension,))


class TurboQuantProd:
    """TurboQuant variant optimized for unbiased inner-product estimation (GPU kernels behind the
    reference API)."""

    def __init__(self, dimension: int, bits: int, *, seed: Optional[int] = None, grid_size: int = 16385,
                 max_iter: int = 200, rotation: Optional[np.ndarray] = None,
                 projection: Optional[np.ndarray] = None):
        if bits < 1:
            raise ValueError("bits must be >= 1")
        self.dimension = int(dimension)
        self.bits = int(bits)
        self.mse = TurboQuantMSE(dimension, max(bits - 1, 1), seed=seed, grid_size=grid_size,
                                 max_iter=max_iter, rotation=rotation)
        if projection is not None:
            self.projection = np.asarray(projection, dtype=np.float32)
        else:
            self.projection = _random_projection_matrix(self.dimension, None if seed is None else seed + 1)
        if self.projection.shape != (self.dimension, self.dimension):
            raise ValueError(
                f"projection must have shape {(self.dimension, self.dimension)}, got {self.projection.shape}"
            )
        self._plans = _PlanSet(self.dimension, self.mse.bits, self.mse.rotation, self.mse.codebook,
                               self.projection)

    def set_kernel_path(self, path: str) -> None:
        self._plans.set_path({"auto": _native.TQ_PATH_AUTO, "exact": _native.TQ_PATH_EXACT,
                              "tensor": _native.TQ_PATH_TENSOR}[path])

    def quantize(self, vectors: Any) -> TurboQuantProdEncoding:
        staged = _stage(vectors, self.dimension)
        pk = self.mse._quantize_staged(staged, self._plans, prod=True)
        return _encoding_from_packed(TurboQuantProdEncoding, pk, staged.prefix)

    def dequantize(self, encoding: TurboQuantProdEncoding):
        pk = _as_packed(encoding, self._plans, need_signs=True)
        out = pk.norms.new_empty(_row_shape(pk.n, encoding.prefix_shape) + (self.dimension,))
        _native.check(_native.load().tq_prod_dequantize(
            self._plans.handle(pk.device), pk.codes.data_ptr(), pk.signs.data_ptr(), pk.residual_norms.data_ptr(),
            pk.norms.data_ptr(), pk.n, out.data_ptr(), _stream_ptr(pk.device)))
        return _in_shape(_deliver(out, pk.kind, pk.plans), tuple(encoding.prefix_shape) + (self.dimension,))

    def attention_score(self, query: Any, encoding: TurboQuantProdEncoding):
        """One query row broadcast over all keys, or one query row per key (_quant.py:334-358)."""
        pk = _as_packed(encoding, self._plans, need_signs=True)
        if (type(query) is np.ndarray and query.size == self.dimension and query.shape[-1:] == (self.dimension,) and query.dtype.kind in "fiub"
                and 1 < pk.n <= _native.TQ_HOST_SCORES and self._plans._path == _native.TQ_PATH_AUTO):
            return self._score_on_host(query, pk, tuple(encoding.prefix_shape))
        staged = _stage_query(query, self.dimension, pk.device)
        q = staged.tensor
        num_codes = pk.n
        q_prefix = staged.prefix
        broadcast = staged.n == 1 and num_codes > 1
        if staged.n == 1:
            q_prefix = tuple(encoding.prefix_shape)
        if not broadcast and staged.n != num_codes:
            raise ValueError(
                f"query batch size {staged.n} does not match encoding batch size {num_codes}"
            )
        lib = _native.load()
        # a short row of scores for a NumPy caller is written straight to page-locked memory (one query: _score_on_host)
        to_host = staged.kind == "numpy" and 4 * num_codes <= _MAPPED_BYTES
        rows = _row_shape(num_codes, q_prefix)
        scores = _torch().empty(rows, dtype=_torch().float32, device="cpu", pin_memory=True) if to_host else pk.norms.new_empty(rows)
        handle = self._plans.handle(pk.device)
        st = _stream_ptr(pk.device)
        if broadcast and self._plans._path == _native.TQ_PATH_AUTO:
            # one query against all keys: the entry point that needs no scratch buffer
            _native.check(lib.tq_score_broadcast(handle, q.data_ptr(), pk.codes.data_ptr(), pk.signs.data_ptr(),
                                                 pk.residual_norms.data_ptr(), pk.norms.data_ptr(), num_codes,
                                                 scores.data_ptr(), st))
        elif broadcast:
            # a forced kernel path: the one-row case of the batched entry point
            need = max(lib.tq_topk_scratch_bytes(handle, 1, 1, num_codes, 0), 16)
            scratch = pk.norms.new_empty((need,), dtype=_torch().uint8)
            _native.check(lib.tq_score_batched(handle, q.data_ptr(), 1, 1, pk.codes.data_ptr(), pk.signs.data_ptr(),
                                               pk.residual_norms.data_ptr(), pk.norms.data_ptr(), num_codes,
                                               scores.data_ptr(), 0, None, None, 0, scratch.data_ptr(), need, st))
        else:
            _native.check(lib.tq_score_pairwise(handle, q.data_ptr(), pk.codes.data_ptr(), pk.signs.data_ptr(),
                                                pk.residual_norms.data_ptr(), pk.norms.data_ptr(), num_codes,
                                                scores.data_ptr(), st))
        if to_host:
            self._plans.check_status(pk.device)      # waits for the stream
            return _in_shape(scores.clone().numpy(), q_prefix)
        return _in_shape(_deliver(scores, staged.kind, self._plans), q_prefix)

    def _score_on_host(self, query: np.ndarray, pk: _Packed, shape):
        """One NumPy query against a few thousand keys: one call into the library takes the query, waits and returns the scores
        (the same through page-locked torch tensors and a call to wait took 31 us instead of 21, the kernel 3 of them)."""
        q = np.ascontiguousarray(query, dtype=np.float32)
        scores = np.empty(pk.n, dtype=np.float32)
        status = ctypes.c_int64(0)
        _native.check(_native.load().tq_score_host(
            self._plans.handle(pk.device), q.__array_interface__["data"][0], pk.codes.data_ptr(), pk.signs.data_ptr(),
            pk.residual_norms.data_ptr(), pk.norms.data_ptr(), pk.n, scores.__array_interface__["data"][0], ctypes.byref(status),
            _stream_ptr(pk.device)))
        if status.value:
            _PlanSet.refuse(status.value)
        return _in_shape(scores, shape)

    def attention_scores(self, queries: Any, encoding: TurboQuantProdEncoding, *, topk: Optional[int] = None,
                         groups: int = 1, return_matrix: Optional[bool] = None, index_base: int = 0,
                         out: Optional[Tuple[Any, Any]] = None):
        """Score many queries against shared keys in one pass over the packed keys.

        ``queries`` has shape (..., d) and flattens to Q rows; the N keys are split into ``groups``
        equal consecutive blocks and the Q rows into ``groups`` equal blocks; query block g meets
        key block g only (``groups=1``: every query meets every key; larger values give the
        per-sequence / per-head batching of a KV cache).  Row i of the result equals
        ``attention_score(queries[i], keys of its block)``.

        Returns the score matrix of shape (Q, N // groups) when ``topk`` is None; with ``topk=k``
        returns ``(top_scores, top_indices)`` of shape (Q, k), descending, indices counted over
        all N keys plus ``index_base`` (set ``return_matrix=True`` to get the matrix as a third
        element as well).  ``out=(top_scores, top_indices)``: contiguous device tensors of shape (Q, k), float32 and
        int64, that receive the top-k instead of fresh ones (e.g. the send block of ``sharded.TopkExchange``, so
        that the candidates need no repacking before the collective).
        """
        pk = _as_packed(encoding, self._plans, need_signs=True)
        staged = _stage_query(queries, self.dimension, pk.device)
        q, new_empty = staged.tensor, pk.norms.new_empty
        nq, n = staged.n, pk.n
        if groups < 1 or nq % groups or n % groups:
            raise ValueError(f"groups={groups} must divide both the query count {nq} and the key count {n}")
        qpg, kpg = nq // groups, n // groups
        k = int(topk) if topk else 0
        want_matrix = (k == 0) if return_matrix is None else bool(return_matrix)
        if k == 0 and not want_matrix:
            raise ValueError("nothing to compute: no top-k requested and return_matrix is False")
        torch = _torch()
        lib = _native.load()
        handle = self._plans.handle(pk.device)
        scores = new_empty((nq, kpg)) if want_matrix else None
        if out is not None and k:
            top_s, top_i = out
            if (tuple(top_s.shape) != (nq, k) or tuple(top_i.shape) != (nq, k) or top_s.dtype != torch.float32
                    or top_i.dtype != torch.int64 or not top_s.is_contiguous() or not top_i.is_contiguous()
                    or top_s.device != pk.device or top_i.device != pk.device):
                raise ValueError(f"out must be contiguous float32 / int64 tensors of shape ({nq}, {k}) on {pk.device}")
        else:
            top_s = new_empty((nq, k)) if k else None
            top_i = new_empty((nq, k), dtype=torch.int64) if k else None
        need = max(lib.tq_topk_scratch_bytes(handle, groups, qpg, kpg, k), 16)
        scratch = new_empty((need,), dtype=torch.uint8)
        _native.check(lib.tq_score_batched(handle, q.data_ptr(), groups, qpg, pk.codes.data_ptr(), pk.signs.data_ptr(),
                                           pk.residual_norms.data_ptr(), pk.norms.data_ptr(), kpg, _ptr(scores), k,
                                           _ptr(top_s), _ptr(top_i), int(index_base), scratch.data_ptr(), need,
                                           _stream_ptr(pk.device)))
        if k == 0:
            return _deliver(scores, staged.kind, self._plans)
        result = (_deliver(top_s, staged.kind, self._plans), _deliver(top_i, staged.kind))
        return result + (_deliver(scores, staged.kind),) if want_matrix else result


def turboquant_mse(vectors: Any, bits: int, *, seed: Optional[int] = None) -> Tuple[TurboQuantMSE, TurboQuantMSEEncoding]:
    """Convenience helper that instantiates and applies `TurboQuantMSE`."""
    array = _to_array(vectors)
    quantizer = TurboQuantMSE(array.shape[-1], bits, seed=seed)
    return quantizer, quantizer.quantize(vectors)


def turboquant_prod(vectors: Any, bits: int, *, seed: Optional[int] = None) -> Tuple[TurboQuantProd, TurboQuantProdEncoding]:
    """Convenience helper that instantiates and applies `TurboQuantProd`."""
    array = _to_array(vectors)
    quantizer = TurboQuantProd(array.shape[-1], bits, seed=seed)
    return quantizer, quantizer.quantize(vectors)
