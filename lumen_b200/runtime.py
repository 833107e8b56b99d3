"""Host-side handles over the C ABI: fused kernels compiled from fusion bodies, GEMM, attention, scatter-add, launched
on device memory the caller holds. Tensors are duck-typed: the backend's own `lumen_b200.device.Tensor`, or any array
of another framework that answers `data_ptr()`, `shape`, `stride()` and `dtype` (a harness may pass torch CUDA
tensors; torch is never imported by this module unless the caller already did). Every kernel that runs is
liblumen_b200's."""

from __future__ import annotations

import ctypes
import math
import sys
import threading
from collections import OrderedDict

from lumen_b200 import _lib
from lumen_b200.graph import Graph


class _TorchDtypes(dict):
    """dtype name -> torch dtype, filled on first use so that importing this module does not import torch."""

    def __missing__(self, key):
        import torch

        self.update({
            "bool": torch.bool, "int8": torch.int8, "int16": torch.int16, "int32": torch.int32, "int64": torch.int64,
            "uint8": torch.uint8, "uint16": torch.uint16, "uint32": torch.uint32, "uint64": torch.uint64,
            "float16": torch.float16, "bfloat16": torch.bfloat16, "float32": torch.float32, "float64": torch.float64,
        })  # fmt: skip
        return dict.__getitem__(self, key)


TORCH_DTYPES = _TorchDtypes()


_names: dict = {}  # dtype object -> lumen dtype name, as they are met


def dtype_name(dtype) -> str:
    """The lumen dtype name of a tensor's `dtype` attribute (a name already, or another framework's dtype object)."""
    if isinstance(dtype, str):
        return dtype
    name = _names.get(dtype)
    if name is None:
        name = str(dtype).rsplit(".", 1)[-1]  # "torch.bfloat16" -> "bfloat16"
        if name not in _lib.DTYPE_CODES:
            raise TypeError(f"no lumen dtype for {dtype!r}")
        _names[dtype] = name
    return name


_cuda_seen = False


def require_cuda() -> None:
    global _cuda_seen
    if not _cuda_seen:  # the devices of a process do not go away
        if _lib.lib().lb_device_count() <= 0:
            raise RuntimeError("lumen_b200 runs on a B200 GPU only: no CUDA device is available and there is no CPU fallback")
        _cuda_seen = True


def desc(t) -> _lib.LbTensor:
    """The lb_tensor descriptor of a device tensor (shape, element strides, data pointer)."""
    if not getattr(t, "is_cuda", True):
        raise ValueError("expected a CUDA tensor")
    return _lib.strided(t.data_ptr(), dtype_name(t.dtype), t.shape, t.stride())


_current = [0]


def set_current_stream(stream) -> None:
    """The stream launches go to when none is given and torch is not in the process (a `lumen_b200.device.Stream`)."""
    _current[0] = getattr(stream, "handle", stream) or 0


def current_stream() -> int:
    """The caller's current stream: torch's when the process uses torch (a harness), else the one set with
    `set_current_stream` (the legacy default stream by default)."""
    if _current[0] == 0:
        torch = sys.modules.get("torch")
        if torch is not None and torch.cuda.is_initialized():
            raw = getattr(torch._C, "_cuda_getCurrentRawStream", None)  # the handle without a Stream object around it
            return raw(torch.cuda.current_device()) if raw is not None else torch.cuda.current_stream().cuda_stream
    return _current[0]


def _stream(stream) -> int:
    return (current_stream() if stream is None else getattr(stream, "handle", stream)) or 0


class Fusion:
    """One generated kernel for a fusion body (`lb_fusion_compile` / `lb_fusion_launch`)."""

    def __init__(self, body: Graph | str):
        text = body if isinstance(body, str) else body.to_text()
        handle = ctypes.c_void_p()
        _lib.check(_lib.lib().lb_fusion_compile(text.encode(), ctypes.byref(handle)))
        self.handle = handle
        self.n_inputs = _lib.lib().lb_fusion_num_inputs(handle)
        self.n_outputs = _lib.lib().lb_fusion_num_outputs(handle)
        self.scratch_bytes = _lib.lib().lb_fusion_scratch_bytes(handle)
        self.body = body if isinstance(body, Graph) else None

    @property
    def source(self) -> str:
        return _lib.lib().lb_fusion_source(self.handle).decode()

    def launch_raw(self, descs, scratch_ptr=None, stream=None) -> None:
        arr = (_lib.LbTensor * len(descs))(*descs)
        _lib.check(
            _lib.lib().lb_fusion_launch(
                self.handle, arr, len(descs), scratch_ptr, current_stream() if stream is None else stream
            )
        )

    def __call__(self, *inputs, out=None, stream=None):
        """Runs the kernel on CUDA tensors; allocates the outputs unless `out` gives them."""
        require_cuda()
        if self.body is None:
            raise RuntimeError("calling a Fusion built from text needs explicit outputs: use launch_raw")
        if out is None:
            out = [_empty_like_input(inputs[0], self.body.types[v].shape, self.body.types[v].dtype) for v in self.body.outputs]
        # partial sums between the call's two kernels: another call must not meet them, on whatever stream, thread or device
        scratch = _workspace(inputs[0], (self.scratch_bytes,), "uint8", stream) if self.scratch_bytes else None
        self.launch_raw([desc(t) for t in (*inputs, *out)], scratch.data_ptr() if scratch is not None else None, stream)
        return out


_regions: dict = {}  # device -> its regions, as they were reserved


def _empty_like_input(like, shape, dtype: str):
    """A new dense device tensor of `shape`/`dtype` in the framework `like` comes from: torch for a torch tensor (the
    harness's convenience), else the backend's own regions of the current device (grown in 256 MiB reservations)."""
    if type(like).__module__.startswith("torch"):
        torch = sys.modules["torch"]
        if type(like) is torch.Tensor:  # 1.5 and 2.0 us a tensor, where `empty` takes 2.4 to read its arguments
            if like.shape == shape:
                return torch.empty_like(like, dtype=TORCH_DTYPES[dtype], memory_format=torch.contiguous_format)
            return like.new_empty(shape, dtype=TORCH_DTYPES[dtype])
        return torch.empty(shape, dtype=TORCH_DTYPES[dtype], device=like.device)
    from lumen_b200.device import ITEMSIZE, Region, current_device

    nbytes = max(math.prod(shape) * ITEMSIZE[dtype], 1)
    regions = _regions.setdefault(current_device(), [])
    for region in regions:
        try:
            return region.empty(shape, dtype)
        except _lib.LumenError:
            continue
    region = Region(max(nbytes + 4096, 256 << 20))
    regions.append(region)
    return region.empty(shape, dtype)


_workspaces: OrderedDict = OrderedDict()  # (device, stream) -> region, the latest used last
_workspaces_lock = threading.Lock()
_WORKSPACE_STREAMS = 8


def _workspace(like, shape, dtype: str, stream):
    """Memory of one call on `stream`, which may be dropped as soon as the call's kernels are queued: what the memory is given to next
    is queued on the same stream. From torch's allocator with `stream` current for a torch tensor, else from a region that serves
    this stream of the current device alone; the regions of the eight latest streams are kept (freeing one waits for its work)."""
    if type(like).__module__.startswith("torch"):
        if stream is None and _current[0] == 0:  # torch's current stream
            return _empty_like_input(like, shape, dtype)
        torch, handle = sys.modules["torch"], _stream(stream)
        with torch.cuda.stream(torch.cuda.ExternalStream(handle, like.device) if handle else torch.cuda.default_stream(like.device)):
            return _empty_like_input(like, shape, dtype)
    from lumen_b200.device import ITEMSIZE, Region, current_device

    key = (current_device(), _stream(stream))
    with _workspaces_lock:
        if key in _workspaces:
            _workspaces.move_to_end(key)
            try:
                return _workspaces[key].empty(shape, dtype)
            except _lib.LumenError:  # too small, or in use by other threads' calls: one that holds all of it takes its place
                live = _workspaces[key].stats()["live_bytes"]
        else:
            live = 0
        region = Region(max(live + math.prod(shape) * ITEMSIZE[dtype] + 4096, 32 << 20))
        work = region.empty(shape, dtype)  # (reserves the memory: a region that cannot be had takes no place)
        _workspaces[key] = region
        while len(_workspaces) > _WORKSPACE_STREAMS:
            _workspaces.popitem(last=False)
        return work


GEMM_KERNELS = {"auto": 0, "tcgen05": 1, "simt": 2, "tcgen05_1cta": 3}
EPILOGUES = {None: 0, "none": 0, "relu": 1, "add": 2, "mask_positive": 3}


def gemm(a, b, out, epilogue=None, kernel="auto", stream=None, scratch=None, aux=None):
    """`out[.., M, N] = a[.., M, K] @ b[.., K, N]` with float32 accumulation through `lb_gemm`. `a` and `b` may be
    transposed views (any unit-stride major); `out` is float32 or the operands' dtype, row-major. `scratch` (a
    uint8 tensor of `gemm_scratch_bytes` bytes) lets few-tile, long-K problems split K. Epilogues: "relu";
    "add" (`round(product) + aux`) and "mask_positive" (`aux > 0 ? round(product) : 0`) with `aux` shaped like `out`.
    Bit-identical from call to call; the same rows in a larger product may differ in the last bit (another number of K
    ranges, which depends on every dimension)."""
    require_cuda()
    scratch_ptr, scratch_bytes = (scratch.data_ptr(), scratch.numel() * scratch.element_size()) if scratch is not None else (0, 0)
    _lib.host().gemm(a, b, out, aux, EPILOGUES[epilogue], GEMM_KERNELS[kernel], scratch_ptr, scratch_bytes, _stream(stream))
    return out


def device_status() -> None:
    """Synchronises and raises if a kernel's bounded wait gave up (`lb_device_status`)."""
    _lib.check(_lib.lib().lb_device_status())


class _Torch:
    """What calls on plain torch tensors take from torch, looked up once: the lookups on the way to `_empty_like_input`, `_workspace` and
    `_stream` cost the host a microsecond a tensor, in front of kernels that take three."""

    tensor = None  # torch.Tensor, once such a tensor has been met

    @classmethod
    def takes(cls, t, stream) -> bool:
        """Whether `t` is a plain torch tensor and the call is for torch's current stream."""
        if cls.tensor is None and type(t).__module__.startswith("torch"):
            torch = sys.modules["torch"]
            if not hasattr(torch._C, "_cuda_getCurrentRawStream"):
                return False
            cls.empty_like, cls.dense, cls.float32 = torch.empty_like, torch.contiguous_format, torch.float32
            cls.raw_stream, cls.device, cls.tensor = torch._C._cuda_getCurrentRawStream, torch._C._cuda_getDevice, torch.Tensor
        return type(t) is cls.tensor and stream is None and _current[0] == 0 and t.is_cuda

    @classmethod
    def like(cls, t):
        return cls.empty_like(t, memory_format=cls.dense)

    @classmethod
    def stream(cls) -> int:
        return cls.raw_stream(cls.device())


def attention_forward(q, k, v, scale=None, causal=False, out=None, lse=None, stream=None):
    """Flash attention forward through `lb_attention_fwd`: `q` [B, Sq, N, H], `k`/`v` [B, Sk, Nkv, H] bfloat16 views;
    returns `(o, lse)` with `o` [B, Sq, N, H] bfloat16 and `lse` [B, N, Sq] float32. Bit-identical from call to call; the
    same sequence in another batch may differ by a rounding of the probabilities to bfloat16 (another kernel, or another
    number of key ranges when few queries meet many keys)."""
    require_cuda()
    b, sq, n, h = q.shape
    sk = k.shape[1]
    if out is None and lse is None and _Torch.takes(q, stream):
        out, lse, handle = _Torch.like(q), q.new_empty((b, n, sq), dtype=_Torch.float32), _Torch.stream()
    else:
        if out is None:
            out = _empty_like_input(q, tuple(q.shape), dtype_name(q.dtype))
        if lse is None:
            lse = _empty_like_input(q, (b, n, sq), "float32")
        handle = _stream(stream)
    _lib.host().attention_fwd(float(scale if scale is not None else h**-0.5), bool(causal), sk - sq, q, k, v, out, lse, handle)
    return out, lse


# What the backward takes for dS whatever memory there is, and at most from a region, which is kept for its stream.
_SMALL_SCORES, _KEPT_SCORES = 64 << 20, 256 << 20


def _out_of_memory(error: RuntimeError) -> bool:
    if isinstance(error, _lib.LumenError):
        return "out of memory" in str(error)
    torch = sys.modules.get("torch")
    return torch is not None and isinstance(error, torch.OutOfMemoryError)


def _memory_is_short(t) -> bool:
    """Whether a request to torch's allocator for memory of `t`'s device has failed before: another one that does not fit would wait for the
    GPU and empty the allocator's cache once more. (10 us.)"""
    try:
        stats = sys.modules["torch"].cuda.memory_stats_as_nested_dict(t.device)
    except RuntimeError:  # an allocator that does not count
        return True
    return stats.get("num_alloc_retries", 0) + stats.get("num_ooms", 0) > 0


def _scores(q, nbytes: int, stream):
    """Memory for the dS that the backward hands on, or None where that may cost more than it gives."""
    if type(q).__module__.startswith("torch"):
        if nbytes > _SMALL_SCORES and _memory_is_short(q):
            return None
    elif nbytes > _KEPT_SCORES:
        return None
    try:
        return _workspace(q, (nbytes,), "uint8", stream)
    except RuntimeError as error:
        if not _out_of_memory(error):
            raise
        return None


def attention_backward(q, k, v, o, d_o, lse, scale=None, causal=False, delta=None, stream=None, deterministic=True, max_scratch=None):
    """Flash attention backward; returns `(dq, dk, dv)` shaped like `q`, `k`, `v`. `deterministic` (the default here)
    runs `lb_attention_bwd_scratch`, the dK/dV + dQ kernel pair that is bit-identical from run to run; without it
    `lb_attention_bwd_atomic` runs the reference backend's default mode, one kernel adding dQ atomically into a float32
    accumulator, at head dim 64, and the same pair elsewhere. At head dim 128 the pair hands dS on in memory of the call's, up to 4.5 GiB
    or `max_scratch` bytes (0: none), where there is such memory; the results are the same either way."""
    require_cuda()
    b, sq, n, h = q.shape
    sk = k.shape[1]
    plain = _Torch.takes(q, stream) and type(k) is type(v) is _Torch.tensor
    if plain:
        dq, dk, dv, handle = _Torch.like(q), _Torch.like(k), _Torch.like(v), _Torch.stream()
        if delta is None:
            delta = q.new_empty((b, n, sq), dtype=_Torch.float32)
    else:
        dq, dk, dv = (_empty_like_input(t, tuple(t.shape), dtype_name(t.dtype)) for t in (q, k, v))
        if delta is None:
            delta = _workspace(q, (b, n, sq), "float32", stream)
        handle = _stream(stream)
    dq_accum = _workspace(q, (b, sq, n, h), "float32", stream) if h == 64 and not deterministic else None
    scale, causal = float(scale if scale is not None else h**-0.5), bool(causal)
    nbytes = _lib.host().attention_bwd_scratch_bytes(scale, causal, sk - sq, q, k) if h == 128 else 0
    if max_scratch is not None:
        nbytes = max(0, min(nbytes, max_scratch))
    scores = _scores(q, nbytes, stream) if nbytes else None
    pointer, nbytes = (0, 0) if scores is None else (scores.data_ptr(), nbytes)
    _lib.host().attention_bwd(scale, causal, sk - sq, q, k, v, o, d_o, lse, delta, dq_accum, dq, dk, dv, pointer, nbytes, handle)
    return dq, dk, dv


def gemm_scratch_bytes(m: int, n: int, k: int, batch: int = 1) -> int:
    """Bytes of scratch with which `gemm` splits K for this problem (0: it would not split)."""
    return _lib.lib().lb_gemm_scratch_bytes(m, n, k, batch)


def scatter_add_rows(x, ids, updates, deterministic=True, stream=None):
    """`x` `[rows, width]` with `updates[t]` added into row `ids[t]` (clamped into range), through
    `lb_scatter_add_rows`. Deterministic form: a row hit more than once adds its updates in update order, rounding
    after each add, like the reference interpreter; otherwise float32 atomics in arrival order and one rounding."""
    require_cuda()
    lib = _lib.lib()
    lib.lb_scatter_add_scratch_bytes.argtypes = [ctypes.c_int64, ctypes.c_int64, ctypes.c_int64, ctypes.c_int]
    lib.lb_scatter_add_scratch_bytes.restype = ctypes.c_size_t
    T = ctypes.POINTER(_lib.LbTensor)
    lib.lb_scatter_add_rows.argtypes = [T, T, T, T, ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int, ctypes.c_void_p]
    rows, width = x.shape
    nbytes = lib.lb_scatter_add_scratch_bytes(rows, width, ids.numel(), int(deterministic))
    scratch = _workspace(x, (max(nbytes, 4),), "uint8", stream)
    out = _empty_like_input(x, tuple(x.shape), dtype_name(x.dtype))
    updates = updates.reshape(-1, width)  # held until the kernels are queued: a view, or a copy of one with other strides
    dx, di, du, do = desc(x), desc(ids), desc(updates), desc(out)
    _lib.check(lib.lb_scatter_add_rows(ctypes.byref(dx), ctypes.byref(di), ctypes.byref(du), ctypes.byref(do), scratch.data_ptr(),
                                       nbytes, int(deterministic), current_stream() if stream is None else stream))
    return out
