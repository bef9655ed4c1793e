"""ctypes binding of ``libq4b200.so`` (the C ABI declared in ``include/q4b200.h``).

The library is loaded on first use.  There is no fallback: if it is missing and cannot be
built, or a call returns an error code, a ``RuntimeError`` carrying the library's own message
is raised.
"""
from __future__ import annotations

import ctypes
import os
import threading
import warnings
from ctypes import c_char_p, c_int, c_longlong, c_size_t, c_uint, c_ulonglong, c_void_p

import torch

_PKG = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(_PKG, "libq4b200.so")

Q4_F16, Q4_F32 = 0, 1
GEMV_ACCUMULATE, GEMV_ACT_ORDER, GEMV_V1, GEMV_WRITTEN = 1, 2, 4, 8

_lib = None
_lock = threading.Lock()

# name -> (restype, argtypes); mirrors include/q4b200.h one to one
_SIGNATURES = {
    "q4_version": (c_int, []),
    "q4_last_error_string": (c_char_p, []),
    "q4_recons_v2": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_void_p]),
    "q4_recons_v1": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_void_p]),
    "q2_recons_v2": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_void_p]),
    "q4_gemv_workspace_bytes": (c_size_t, [c_int, c_int, c_int]),
    "q4_layer_create": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int]),
    "q4_layer_gemv": (c_int, [c_void_p, c_void_p, c_void_p, c_int, c_void_p, c_size_t, c_void_p]),
    "q4_layer_destroy": (None, [c_void_p]),
    "q4_layer_set_next": (c_int, [c_void_p, c_void_p]),
    "q4_gemv_set_trace": (c_int, [c_void_p]),
    "q4_gemm_set_trace": (c_int, [c_void_p]),
    "q4_gemm_set_variant": (c_int, [c_int]),
    "q4_gemv_set_variant": (c_int, [c_int]),
    "q4_gemv_static_max_bytes": (c_size_t, []),
    "q4_gemv_static": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,
                               c_int, c_int, c_int, c_int, c_int, c_int, c_uint, c_void_p]),
    "q4_gemm_fwd": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,
                            c_int, c_int, c_int, c_int, c_int, c_void_p, c_size_t, c_void_p]),
    "q4_gemm_bwd": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,
                            c_int, c_int, c_int, c_int, c_int, c_void_p, c_size_t, c_void_p]),
    "q4_clear": (c_int, [c_void_p, c_size_t, c_void_p]),
    "q4_capture_id": (c_int, [c_void_p, ctypes.POINTER(c_ulonglong)]),
    "q4_gemm_plan": (c_int, [c_int, c_int, c_int, c_int, c_int, c_int, c_int, c_size_t, c_void_p, c_void_p]),
    "q4_gemm_workspace_bytes": (c_size_t, [c_int, c_int, c_int]),
    "q4_zero_term_table": (c_int, [c_void_p, c_void_p, c_void_p, c_int, c_int, c_void_p]),
    "q4_gemm_fwd_residual": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,
                                     c_void_p, c_int, c_int, c_int, c_int, c_int, c_int, c_void_p, c_size_t, c_void_p]),
    "q4_gemm_fwd_v1": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_void_p,
                               c_size_t, c_void_p]),
    "q4_gemm_fwd_table": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,
                                  c_int, c_int, c_int, c_int, c_int, c_void_p, c_size_t, c_void_p]),
    "q4_gemm_bwd_table": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int,
                                  c_int, c_int, c_int, c_int, c_void_p, c_size_t, c_void_p]),
    "q4_gemm_fwd_swiglu": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int,
                                   c_int, c_int, c_void_p, c_size_t, c_void_p]),
    "q4_rmsnorm_fwd": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, ctypes.c_float, c_void_p]),
    "q4_rmsnorm_bwd": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_void_p]),
    "q4_swiglu_fwd": (c_int, [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_void_p]),
    "q4_swiglu_bwd": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_void_p]),
    "q4_rope": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int, c_int, c_void_p]),
    "q4_lora_project": (c_int, [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, ctypes.c_float, c_void_p]),
    "q4_cast16": (c_int, [c_void_p, c_void_p, c_size_t, c_int, c_void_p]),
    "q4_causal_loss_fwd": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_longlong, c_int, c_void_p]),
    "q4_causal_loss_fwd_keep": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_longlong,
                                        c_int, c_void_p]),
    "q4_causal_loss_bwd": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_longlong, c_int, c_void_p]),
    "q4_lora_grads": (c_int, [c_void_p, c_void_p, c_void_p, c_int, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_void_p]),
    "q4_adamw_flat": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_size_t, ctypes.c_float, ctypes.c_float, ctypes.c_float,
                              ctypes.c_float, ctypes.c_float, ctypes.c_float, c_void_p, ctypes.c_float, ctypes.c_float, c_int, c_void_p, c_void_p]),
    "q4_device_status": (c_int, [ctypes.POINTER(c_uint)]),
    "q4_gemv_status": (c_int, [c_void_p, c_size_t, ctypes.POINTER(c_uint)]),
    "q4_gemv_device_status": (c_int, [c_void_p]),
    "q4_gemv_static_status": (c_int, [ctypes.POINTER(c_uint)]),
    "q4_gemv": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,
                        c_int, c_int, c_int, c_int, c_int, c_int, c_uint, c_void_p, c_size_t, c_void_p]),
}


def exported_symbols():
    return sorted(_SIGNATURES)


def lib() -> ctypes.CDLL:
    """The loaded library (built in-tree on first use when nvcc is present)."""
    global _lib
    if _lib is not None:
        return _lib
    with _lock:
        if _lib is not None:
            return _lib
        if not os.path.exists(LIB_PATH):
            from . import build as _build
            _build.build()
        handle = ctypes.CDLL(LIB_PATH)
        for name, (res, args) in _SIGNATURES.items():
            fn = getattr(handle, name)          # AttributeError here = header and library disagree
            fn.restype, fn.argtypes = res, args
        _lib = handle
    return _lib


_layer_gemv_call = None


def layer_gemv_call():
    """``q4_layer_gemv`` as a callable of seven Python ints that returns the C return code: the ``_q4call``
    extension module (built in-tree with the C compiler on first use), bound to the loaded library.  It
    makes the same foreign call as the ctypes binding without ctypes' per-argument conversion."""
    global _layer_gemv_call
    if _layer_gemv_call is not None:
        return _layer_gemv_call
    handle = lib()
    with _lock:
        if _layer_gemv_call is None:
            from . import build as _build
            _build.build_call()
            from . import _q4call
            _q4call.bind(ctypes.cast(handle.q4_layer_gemv, c_void_p).value)
            _layer_gemv_call = _q4call.layer_gemv
    return _layer_gemv_call


class _NoTorchCall:
    """In the place of ``_q4torch`` where it cannot be built or loaded: takes no operands, so that every product goes through
    the ctypes binding, to the same kernels."""
    @staticmethod
    def gemv(*_):
        return None

    gemm = gemm_v1 = swiglu = gemv


_torch_call = None


def torch_call():
    """The ``_q4torch`` module (built in-tree on first use, and again when its sources or torch have changed), bound to the
    loaded library: products on torch tensors as one native call each.  Its functions return ``None`` for operands they do
    not take.  Without a C++ compiler or torch's headers, say, the reason is given once and the stand-in above serves."""
    global _torch_call
    if _torch_call is not None:
        return _torch_call
    handle = lib()
    with _lock:
        if _torch_call is None:
            try:
                from . import build as _build
                _build.build_torch_call()
                from . import _q4torch
                _q4torch.bind(*(ctypes.cast(getattr(handle, name), c_void_p).value for name in (
                    "q4_gemv", "q4_gemm_fwd_residual", "q4_gemm_bwd_table", "q4_gemm_bwd", "q4_swiglu_fwd", "q4_last_error_string", "q4_gemm_fwd_v1")))
                _torch_call = _q4torch
            except Exception as e:
                warnings.warn(f"q4b200: the native module for torch tensors is not available ({type(e).__name__}: {e}); "
                              "products go through the ctypes binding, at a higher cost per call")
                _torch_call = _NoTorchCall
    return _torch_call


_transforms, _tracing, _forward_ad = torch._C._functorch.peek_interpreter_stack, torch._C._get_tracing_state, torch.autograd.forward_ad


def nobody_watches() -> bool:
    """No function transform (vmap, grad), forward-mode level or tracer is active that would have to see the operations of
    this call."""
    return _transforms() is None and _forward_ad._current_level < 0 and _tracing() is None


def opaque_call_ok(x) -> bool:
    """A call that torch does not see into may stand for operations on ``x``: a plain GPU tensor that nothing
    differentiates, batches or traces through this call."""
    return x.is_cuda and type(x) is torch.Tensor and not (torch.is_grad_enabled() and x.requires_grad) and nobody_watches()


def check(code: int, what: str) -> None:
    if code != 0:
        msg = lib().q4_last_error_string().decode("utf-8", "replace")
        raise RuntimeError(f"q4b200 {what} failed ({code}): {msg}")


def ptr(t) -> int | None:
    return None if t is None else t.data_ptr()


def stream_of(t: torch.Tensor) -> int:
    return torch.cuda.current_stream(t.device).cuda_stream


def require_cuda(*tensors) -> torch.device:
    """All tensors must live on one CUDA device and be contiguous; returns that device."""
    dev = None
    for t in tensors:
        if t is None:
            continue
        if not t.is_cuda:
            raise RuntimeError("q4b200: tensors must be CUDA tensors (there is no CPU path)")
        if not t.is_contiguous():
            raise RuntimeError("q4b200: tensors must be contiguous")
        if dev is None:
            dev = t.device
        elif t.device != dev:
            raise RuntimeError(f"q4b200: tensors on different devices ({dev} vs {t.device})")
    return dev


class on_device:
    """Make ``dev`` the current CUDA device for the duration of a call; free when it already is."""
    __slots__ = ("dev", "prev")

    def __init__(self, dev: torch.device):
        self.dev = dev.index if dev.index is not None else torch.cuda.current_device()
        self.prev = -1

    def __enter__(self):
        cur = torch.cuda.current_device()
        if cur != self.dev:
            self.prev = cur
            torch.cuda.set_device(self.dev)
        return self

    def __exit__(self, *exc):
        if self.prev >= 0:
            torch.cuda.set_device(self.prev)
        return False


def dtype_code(dt: torch.dtype) -> int:
    if dt == torch.float16:
        return Q4_F16
    if dt == torch.float32:
        return Q4_F32
    raise RuntimeError(f"q4b200: unsupported dtype {dt} (float16 or float32)")


_workspaces: dict = {}
_WS_BYTES = 4 << 20          # covers q4_gemv_workspace_bytes() of every shape the decode kernels accept
_DECODE_WS_HEAD = 131072     # what the decode kernels need zero before the first call and leave zero
_gemm_workspaces: dict = {}
_GEMM_WS_HEAD = 65536        # arrival counters: zero before the first call, left zero by every kernel

# Workspaces of stream captures: (device index, stream handle) and, for decode, the same with "decode" -> (id of the
# capture, its workspaces, the newest last).
# A graph holds the addresses of its products' workspaces for as long as it lives, so every capture has its own, from the memory
# of its graph and cleared by it.  (The stream's own one makes way for a larger one; first asked for inside a capture it was cleared
# by that graph's replay alone; and torch captures every graph on one stream unless told otherwise, so that two graphs
# replayed on two streams counted their arrivals in one place.)  A graph is larger by them: 4 MiB with decode products, 24 to 42
# with fused ones.  They are only held here for the next product of the same capture, and let go by the first eager product after
# it: an eager call of another thread in the middle of a capture costs that capture a second workspace, nothing else.
_capture_workspaces: dict = {}


def _of_capture(key, capture: int, nbytes: int, head: int, device: torch.device, stream_handle: int) -> torch.Tensor:
    held = _capture_workspaces.get(key)
    if held is None or held[0] != capture:
        held = _capture_workspaces[key] = (capture, [])
    if not held[1] or held[1][-1].numel() < nbytes:
        ws = torch.empty(nbytes, dtype=torch.uint8, device=device)
        if device.type == "cuda":
            check(lib().q4_clear(ws.data_ptr(), head, stream_handle), "clear")
        else:
            ws[:head].zero_()
        held[1].append(ws)
        return ws
    return held[1][-1]


def capture_id(stream_handle: int) -> int:
    """The number of the capture that ``stream_handle`` is part of (no two captures of a process share one)."""
    out = ctypes.c_ulonglong(0)
    check(lib().q4_capture_id(stream_handle, ctypes.byref(out)), "capture_id")
    return out.value


def _capture_of(stream_handle: int) -> int:
    """0 outside a capture; the legacy default stream (handle 0) cannot be captured."""
    return capture_id(stream_handle) if stream_handle and torch.cuda.is_current_stream_capturing() else 0


def workspace_for(device: torch.device, stream_handle: int) -> torch.Tensor:
    """The decode workspace of one (device, stream): allocated zeroed on first use, then reused; a capture has its own."""
    key = (device.index, stream_handle)
    capture = _capture_of(stream_handle)
    if capture:
        return _of_capture(key + ("decode",), capture, _WS_BYTES, _DECODE_WS_HEAD, device, stream_handle)
    _capture_workspaces.clear()
    ws = _workspaces.get(key)
    if ws is None:
        ws = torch.zeros(_WS_BYTES, dtype=torch.uint8, device=device)
        _workspaces[key] = ws
    return ws


def gemm_workspace_for(device: torch.device, stream_handle: int, nbytes: int) -> torch.Tensor:
    """Scratch of the fused GEMM for one (device, stream): zeroed when (re)allocated, only ever grows; a capture has its own.
    The kernels leave its counter head zero, so calls ordered on the stream can share it."""
    key = (device.index, stream_handle)
    capture = _capture_of(stream_handle)
    if capture:
        return _of_capture(key, capture, max(nbytes, 24 << 20), _GEMM_WS_HEAD, device, stream_handle)
    _capture_workspaces.clear()
    ws = _gemm_workspaces.get(key)
    if ws is None or ws.numel() < nbytes:
        ws = torch.zeros(max(nbytes, 24 << 20), dtype=torch.uint8, device=device)
        _gemm_workspaces[key] = ws
    return ws


def workspace(device: torch.device, nbytes: int) -> torch.Tensor:
    """The decode workspace of the current stream, grown to ``nbytes`` where it is smaller (and cleared then)."""
    stream = torch.cuda.current_stream(device).cuda_stream
    ws = workspace_for(device, stream)
    if ws.numel() < nbytes:
        ws = torch.zeros(nbytes, dtype=torch.uint8, device=device)
        if not _capture_of(stream):
            _workspaces[(device.index, stream)] = ws
    return ws
