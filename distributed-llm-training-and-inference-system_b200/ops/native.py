"""ctypes binding to ``lib/libllmctl_b200.so`` (C ABI in ``include/llmctl_b200.h``).

The library is plain nvcc output with no torch dependency; tensors cross the boundary as raw device
pointers plus the current CUDA stream.  Loading is lazy.  On a machine with a GPU the library MUST be
present — ``lib()`` raises instead of letting callers fall back silently.

Reference parity: the reference has no native layer.
"""
from __future__ import annotations

import ctypes
import importlib.util
import threading
import warnings
from pathlib import Path
from typing import Optional

import torch

from ..utils import nvtx as _nvtx

_LIB_DIR = Path(__file__).resolve().parent.parent / "lib"
_LIB_PATH = _LIB_DIR / "libllmctl_b200.so"
_lock = threading.Lock()
_lib: Optional[ctypes.CDLL] = None

_OPS_PATH = _LIB_DIR / "llmctl_ops.so"
_launches = 0


class _NoOps:
    """Stands in for the extension until the kernel library is loaded on a machine with a GPU: takes nothing."""

    def __getattr__(self, name):
        return _nothing

    @staticmethod
    def launches() -> int:
        return 0


def _nothing(*args):
    return None


#: the operators' host side (csrc/torch/ops.cpp): each function returns None for what it does not take
fast = _NoOps()


def __getattr__(name: str):
    # launch_count: number of native kernel launches issued through this module and the extension (bench.py reports it)
    if name == "launch_count":
        return _launches + fast.launches()
    raise AttributeError(name)


def count_launches(n: int) -> None:
    global _launches
    _launches += n

c_void_p, c_int, c_ll, c_float = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float

_SIGNATURES = {
    "llmctl_rmsnorm_fwd": [c_void_p] * 6 + [c_int, c_int, c_float, c_void_p],
    "llmctl_rmsnorm_bwd": [c_void_p] * 8 + [c_int, c_int, c_int, c_int, c_void_p],
    "llmctl_layernorm_fwd": [c_void_p] * 8 + [c_int, c_int, c_float, c_void_p],
    "llmctl_layernorm_bwd": [c_void_p] * 10 + [c_int, c_int, c_int, c_int, c_void_p],
    "llmctl_rope_inplace": [c_void_p, c_ll, c_int, c_int, c_int, c_void_p, c_void_p, c_void_p, c_int, c_float, c_void_p],
    "llmctl_swiglu_fwd": [c_void_p, c_void_p, c_int, c_int, c_ll, c_void_p],
    "llmctl_swiglu_bwd": [c_void_p, c_void_p, c_void_p, c_int, c_int, c_ll, c_void_p],
    "llmctl_adamw_step": [c_void_p] * 4 + [c_int, c_void_p, c_ll] + [c_float] * 8 + [c_void_p, c_void_p],
    "llmctl_sumsq": [c_void_p, c_int, c_ll, c_void_p, c_int, c_void_p, c_int, c_void_p],
    "llmctl_cross_entropy_fwd_bwd": [c_void_p, c_ll, c_void_p, c_void_p, c_void_p, c_int, c_int, c_ll, c_float, c_void_p, c_int, c_void_p],
    "llmctl_cross_entropy_mean": [c_void_p, c_ll, c_void_p, c_void_p, c_int, c_int, c_ll, c_float, c_int, c_void_p, c_void_p],
    "llmctl_cross_entropy_partial": [c_void_p, c_ll, c_void_p, c_void_p, c_int, c_int, c_ll, c_void_p],
    "llmctl_cross_entropy_finalize": [c_void_p, c_ll, c_void_p, c_void_p, c_int, c_int, c_ll, c_ll, c_float, c_void_p, c_void_p],
    "llmctl_gemm_bf16": [c_void_p] * 3 + [c_int] * 3 + [c_ll] * 3 + [c_int] * 6 + [c_void_p],
    "llmctl_gemm_bf16_bgated": [c_void_p] * 3 + [c_int] * 3 + [c_ll] * 3 + [c_int] * 6 + [c_void_p, ctypes.c_uint, c_ll, c_ll, c_void_p],
    "llmctl_gemm_swiglu_bf16": [c_void_p] * 4 + [c_int] * 3 + [c_ll] * 4 + [c_void_p],
    "llmctl_gemm_swiglu_bwd_bf16": [c_void_p] * 4 + [c_int] * 3 + [c_ll] * 3 + [c_void_p],
    "llmctl_gemm_skinny_scratch_elems": [c_int] * 4,
    "llmctl_stream_capture_id": [c_void_p],
    "llmctl_gemm_skinny_bf16": [c_void_p] * 3 + [c_int] * 3 + [c_ll] * 3 + [c_void_p, c_ll, c_void_p, c_int, c_int, c_void_p],
}
# result types by name; int for the rest
_RESULTS: dict = {"llmctl_gemm_skinny_scratch_elems": c_ll, "llmctl_stream_capture_id": ctypes.c_ulonglong}


def library_path() -> Path:
    return _LIB_PATH


def available() -> bool:
    return _LIB_PATH.exists()


def lib() -> ctypes.CDLL:
    """Load (once) and return the kernel library; raise with build instructions if it is missing."""
    global _lib
    if _lib is not None:
        return _lib
    with _lock:
        if _lib is not None:
            return _lib
        if not _LIB_PATH.exists():
            raise RuntimeError(
                f"native kernel library not found at {_LIB_PATH}; run `python build_native.py` "
                "(or __graft_entry__.build()) — refusing to fall back to PyTorch ops on a GPU")
        l = ctypes.CDLL(str(_LIB_PATH), mode=ctypes.RTLD_GLOBAL)
        for name, argtypes in _SIGNATURES.items():
            try:
                fn = getattr(l, name)
            except AttributeError:
                continue
            fn.restype = _RESULTS.get(name, c_int)
            fn.argtypes = argtypes
        if torch.cuda.is_available() and not _nvtx.KERNEL_RANGES:        # ranges around launches are made in `call`
            _load_ops()
        _lib = l
    return _lib


def _load_ops() -> None:
    """Take the operators' host side in C++ into use.  Where there is none for this PyTorch the Python operators launch the same kernels, at 10-50 us
    more of host time each, which is said once."""
    global fast
    try:
        if not _OPS_PATH.exists():
            raise ImportError("not built")
        spec = importlib.util.spec_from_file_location("llmctl_ops", _OPS_PATH)
        ops = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(ops)
    except (ImportError, OSError) as e:
        warnings.warn(f"{_OPS_PATH.name} is not used ({e}): operators take their checks and launches through Python; run `python build_native.py`", RuntimeWarning)
        return
    ops.bind(str(_LIB_PATH), NativeError, check_waits, _buffered_wgrad)
    fast = ops


def _buffered_wgrad(dy, x, w):
    """The gradient of a weight that has a buffer for it, for the extension's nodes."""
    from .functional import _wgrad
    return _wgrad(dy, x, w)


def register_signature(name: str, argtypes: list, restype=c_int) -> None:
    """``restype``: what the entry point returns where that is not a status."""
    _SIGNATURES[name] = argtypes
    _RESULTS[name] = restype
    if _lib is not None:
        try:
            fn = getattr(_lib, name)
            fn.restype = restype
            fn.argtypes = argtypes
        except AttributeError:
            pass


_functions: dict = {}       # entry points of the loaded library by name; the library is loaded once and never replaced


def _function(name: str):
    fn = _functions.get(name)
    if fn is None:
        fn = _functions[name] = getattr(lib(), name)
    return fn


def has_symbol(name: str) -> bool:
    """Whether the kernel library is built and has this entry.  One that is there and does not load raises."""
    if _lib is None and not available():
        return False
    try:
        _function(name)
        return True
    except AttributeError:
        return False


def ptr(t: Optional[torch.Tensor]) -> Optional[int]:
    return None if t is None else t.data_ptr()


_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)
_raw_device = getattr(torch._C, "_cuda_getDevice", None)


def stream_ptr() -> int:
    """Raw handle of the current CUDA stream.  ``torch.cuda.current_stream()`` builds a Stream object through several
    Python layers (~15 us); a training step asks ~500 times, which made tensor-parallel steps host-bound."""
    if _raw_stream is not None and _raw_device is not None:
        return _raw_stream(_raw_device())
    return torch.cuda.current_stream().cuda_stream


_forward_ad = torch.autograd.forward_ad
_interpreter = torch._C._functorch.peek_interpreter_stack
_tracing_state = torch._C._get_tracing_state


class _NoContext:
    """Stands in for an autograd context where nothing is recorded: keeps what the forward sets on it and saves nothing."""
    needs_input_grad = ()

    def save_for_backward(self, *tensors) -> None:
        pass

    def mark_non_differentiable(self, *tensors) -> None:
        pass

    def mark_dirty(self, *tensors) -> None:
        for t in tensors:
            if not t.is_inference():
                torch.autograd.graph.increment_version(t)


def apply(fn, *args):
    """``fn.apply(*args)`` of an autograd function whose forward is one kernel call.  Where no gradient can be recorded the
    forward is called itself: the autograd machinery costs about 10 us, twice the launch (model_logits of 12 layers makes 98 such
    calls).  Forward-mode AD, functorch transforms and tracing still go through ``apply``, which refuses or records them."""
    if torch.is_grad_enabled():
        for a in args:
            if isinstance(a, torch.Tensor) and a.requires_grad:
                return fn.apply(*args)
    if _forward_ad._current_level >= 0 or _interpreter() is not None or _tracing_state() is not None:
        return fn.apply(*args)
    return fn.forward(_NoContext(), *args)


def keep(ctx, *tensors) -> None:
    """``ctx.save_for_backward`` of tensors that a backward will hand to a kernel (``kept``)."""
    ctx.save_for_backward(*tensors)
    ctx.kept_as = tuple(None if t is None else (t.shape, t.dtype, t.device) for t in tensors)


def kept(ctx):
    """``ctx.saved_tensors``.  A hook on saved tensors may give back anything: what has another size, type or device than what was kept is
    refused before a kernel reads it as that."""
    tensors = ctx.saved_tensors
    for t, form in zip(tensors, ctx.kept_as):
        if form is not None and (t.shape, t.dtype, t.device) != form:
            raise RuntimeError(f"a saved tensor came back as {t.dtype} of sizes {list(t.shape)} on {t.device}")
    return tensors


class NativeError(RuntimeError):
    pass


# Kernels whose bounded waits report when they run out (csrc/common/wait_status.h), in the order of their bytes in the host word, with
# the entry points that read and clear their device-side status.
_WAITS = (("flash attention forward", "llmctl_flash_fwd_status"), ("flash attention backward", "llmctl_flash_bwd_status"),
          ("cross-entropy", "llmctl_cross_entropy_status"), ("latent attention", "llmctl_latent_attention_t5_status"))
_wait_word = ctypes.c_uint32(0)         # the library's word once a kernel has been launched
_wait_bound = False


def _bind_waits() -> None:
    global _wait_word, _wait_bound
    register_signature("llmctl_wait_status_word", [], restype=c_void_p)
    address = _function("llmctl_wait_status_word")()
    if address:
        _wait_word = ctypes.c_uint32.from_address(address)
    _wait_bound = True


def check_waits(context: str = "") -> None:
    """Raise ``NativeError`` if a bounded wait of a kernel has run out since the last report: what that launch and those after it computed
    is invalid.  Reads a word of host memory, so it costs nothing, and sees what has finished: call it where the device has been waited for."""
    value = _wait_word.value
    if value:
        _wait_word.value = 0
        names = [name for i, (name, _) in enumerate(_WAITS) if value >> 8 * i & 0xff]
        for _, status in _WAITS:
            if has_symbol(status):
                _function(status)(1)
        raise NativeError(f"a bounded wait ran out in: {', '.join(names)}{(' (' + context + ')') if context else ''}; "
                          "results since the last check are invalid")


#: kernels launched per entry point when it is not exactly one
_KERNELS_PER_CALL = {"llmctl_rmsnorm_bwd": 2, "llmctl_layernorm_bwd": 3, "llmctl_sumsq": 2, "llmctl_rmsnorm_bwd_noalloc": 2,
                     "llmctl_cross_entropy_mean": 3, "llmctl_flash_attn_bwd": 2, "llmctl_rs_sumsq": 2, "llmctl_ag_gemm": 2,
                     "llmctl_comm_watchdog_poll": 0, "llmctl_comm_watchdog_set_timeout_ms": 0}


def call(name: str, *args) -> None:
    """Invoke a C entry point and raise on a non-zero status."""
    global _launches
    if not _wait_bound:
        _bind_waits()
    if _wait_word.value:
        check_waits("found before " + name)
    fn = _functions.get(name) or _function(name)
    if _nvtx.KERNEL_RANGES:
        with _nvtx.nvtx_range(name):
            rc = fn(*args)
    else:
        rc = fn(*args)
    _launches += _KERNELS_PER_CALL.get(name, 1)
    if rc != 0:
        raise NativeError(f"{name} failed with cudaError {rc}")
