"""Host-side operators on torch tensors: thin, allocation-explicit wrappers over the C ABI.

These mirror how the reference reaches an external kernel: destination-passing packed
functions on DLPack tensors (``R.call_tir("b200.q4f16_matmul", (x, wq, scales), out_sinfo)``;
reference: python/tvm/relax/op/base.py:47-91, src/relax/transform/call_tir_rewrite.cc:55-116).
torch is used only for device memory and streams.
"""
from __future__ import annotations

import ctypes
import importlib.util

import torch

from . import _lib, build
from ._lib import B200Error, DLDataType, DLDevice, DLTensor  # noqa: F401


import contextlib


def _stream_ptr(device) -> int:
    if torch.device(device).type != "cuda":
        return 0
    return torch.cuda.current_stream(device).cuda_stream


def _on(device):
    """Makes `device` current for the call; a CPU tensor is passed through so that the library's
    own validation rejects it (there is no host implementation to fall back to)."""
    return torch.cuda.device(device) if torch.device(device).type == "cuda" else contextlib.nullcontext()


_DTYPES = {
    torch.float16: (2, 16),
    torch.float32: (2, 32),
    torch.uint32: (1, 32),
    torch.int32: (0, 32),
    torch.uint8: (1, 8),
}


class _DLView:
    """Keeps the ctypes arrays of a DLTensor view alive."""

    def __init__(self, t: torch.Tensor):
        code, bits = _DTYPES[t.dtype]
        self.shape = (ctypes.c_int64 * t.dim())(*t.shape)
        self.strides = (ctypes.c_int64 * t.dim())(*t.stride())
        if t.is_cuda:
            dev = DLDevice(2, t.device.index if t.device.index is not None else torch.cuda.current_device())
        else:
            dev = DLDevice(1, 0)
        self.tensor = DLTensor(
            ctypes.c_void_p(t.data_ptr()), dev, t.dim(), DLDataType(code, bits, 1),
            ctypes.cast(self.shape, ctypes.POINTER(ctypes.c_int64)),
            ctypes.cast(self.strides, ctypes.POINTER(ctypes.c_int64)), 0,
        )
        self.keep = t

    def ptr(self):
        return ctypes.byref(self.tensor)


def to_dltensor(t: torch.Tensor) -> _DLView:
    return _DLView(t)


LAYOUTS = {"reference": _lib.LAYOUT_REFERENCE, "paired": _lib.LAYOUT_PAIRED}


def _layout_code(layout) -> int:
    if isinstance(layout, str):
        if layout not in LAYOUTS:
            raise ValueError(f"unknown weight layout {layout!r}; one of {sorted(LAYOUTS)}")
        return LAYOUTS[layout]
    return int(layout)


class _option_scope:
    """Sets a process-wide option of the library for the duration of a block."""

    def __init__(self, name: str, value: int):
        self.name, self.value = name, value

    def __enter__(self):
        L = _lib.lib()
        self.saved = L.b200_get_option(self.name.encode())
        _lib.check(L.b200_set_option(self.name.encode(), self.value))

    def __exit__(self, *exc):
        _lib.check(_lib.lib().b200_set_option(self.name.encode(), self.saved))


_F16, _U32 = torch.float16, torch.uint32


def _plain(device, *tensors) -> bool:
    """True when the tensors are contiguous 2-D tensors on the current CUDA device, so that their pointers and shapes
    say all that a DLPack view would."""
    for t in tensors:
        if t.device != device or t.dim() != 2 or not t.is_contiguous():
            return False
    return device.type == "cuda" and torch._C._cuda_getDevice() == device.index


def _matmul_by_pointer(L, x, wq, scales, out, layout) -> bool:
    """The call through the raw-pointer entry point: what the DLPack entry point checks is checked here (a handful of
    attribute reads) instead of being marshalled into four ctypes structures, which took 25 of a call's 30 us.  False:
    nothing has been launched, the DLPack entry point takes the call or names the error."""
    if x.dtype is not _F16 or wq.dtype is not _U32 or scales.dtype is not _F16 or out.dtype is not _F16:
        return False
    device = x.device
    if not _plain(device, x, wq, scales, out):
        return False
    m, k = x.shape
    n = wq.shape[0]
    if k % 32 or wq.shape[1] * 8 != k or scales.shape != (n, k // 32) or out.shape != (m, n):
        return False
    stream = torch._C._cuda_getCurrentRawStream(device.index)
    L.b200_set_stream(stream)
    if layout is None:
        return L.b200_q4f16_matmul(x.data_ptr(), wq.data_ptr(), scales.data_ptr(), out.data_ptr(), m, n, k, stream) == 0
    return L.b200_q4f16_matmul_layout(x.data_ptr(), wq.data_ptr(), scales.data_ptr(), out.data_ptr(), m, n, k,
                                      _layout_code(layout), stream) == 0


def _dequantize_by_pointer(L, wq, scales, out) -> bool:
    """As :func:`_matmul_by_pointer`, for the decode stage alone."""
    if wq.dtype is not _U32 or scales.dtype is not _F16 or out.dtype is not _F16:
        return False
    device = wq.device
    if not _plain(device, wq, scales, out):
        return False
    n, k = wq.shape[0], wq.shape[1] * 8
    if k % 32 or scales.shape != (n, k // 32) or out.shape != (n, k):
        return False
    stream = torch._C._cuda_getCurrentRawStream(device.index)
    L.b200_set_stream(stream)
    return L.b200_q4f16_dequantize(wq.data_ptr(), scales.data_ptr(), out.data_ptr(), n, k, stream) == 0


_native = None      # the extension module, bound to the loaded library; False: not built for this torch (the checks run in Python then)


def _torch_call():
    global _native
    if _native is None:
        path = build.torch_call_path(torch.__version__)
        try:
            spec = importlib.util.spec_from_file_location(__package__ + "._torch_call", path)
            module = importlib.util.module_from_spec(spec)
        except ImportError:                 # (no such file, or one that does not load)
            _native = False
        else:
            L = _lib.lib()
            module.bind(*(ctypes.cast(fn, ctypes.c_void_p).value
                          for fn in (L.b200_set_stream, L.b200_q4f16_matmul, L.b200_q4f16_matmul_layout, L.b200_q4f16_dequantize)))
            _native = module
    return _native


def q4f16_matmul(x: torch.Tensor, wq: torch.Tensor, scales: torch.Tensor, out: torch.Tensor | None = None,
                 family: str = "auto", layout=None) -> torch.Tensor:
    """y[M,N] fp16 = x[M,K] . decode(wq[N,K/8], scales[N,K/32])^T.  Plain contiguous tensors on the current device go
    straight to the raw-pointer entry point (through the extension, or with the same checks in Python); everything else goes
    through the DLPack entry point, which validates it and names the error.  ``family`` = "auto" | "gemv" | "gemm" picks the raw
    entry point of one kernel family instead.  ``layout`` ("reference" | "paired") names the nibble order
    of ``wq`` for this call; None takes the library's option "weights.layout"."""
    if out is None:
        out = torch.empty((x.shape[0], wq.shape[0]), dtype=torch.float16, device=x.device)
    if family == "auto":
        native = _native or _torch_call()
        if native and native.matmul(x, wq, scales, out, -1 if layout is None else _layout_code(layout)):
            return out
    L = _lib.lib()
    if family == "auto":
        if _matmul_by_pointer(L, x, wq, scales, out, layout):
            return out
        with _on(x.device):
            L.b200_set_stream(_stream_ptr(x.device))
            vx, vw, vs, vy = (_DLView(t) for t in (x, wq, scales, out))
            if layout is None:
                _lib.check(L.b200_q4f16_matmul_dl(vx.ptr(), vw.ptr(), vs.ptr(), vy.ptr()))
            else:
                code = _lib.family_with_layout(_lib.FAMILY_AUTO, _layout_code(layout))
                _lib.check(L.b200_q4f16_matmul_dl_family(vx.ptr(), vw.ptr(), vs.ptr(), vy.ptr(), code))
        return out
    fn = {"gemv": L.b200_q4f16_gemv, "gemm": L.b200_q4f16_gemm, "gemm_ws": L.b200_q4f16_gemm_ws,
          "matmul": L.b200_q4f16_matmul}[family]
    M, K = x.shape
    N = wq.shape[0]
    with _on(x.device):
        if layout is None:
            _lib.check(fn(x.data_ptr(), wq.data_ptr(), scales.data_ptr(), out.data_ptr(), M, N, K, _stream_ptr(x.device)))
        else:
            with _option_scope("weights.layout", _layout_code(layout)):
                _lib.check(fn(x.data_ptr(), wq.data_ptr(), scales.data_ptr(), out.data_ptr(), M, N, K, _stream_ptr(x.device)))
    return out


def q4f16_repack(wq: torch.Tensor, layout="paired", out: torch.Tensor | None = None) -> torch.Tensor:
    """The packed words of ``wq`` (reference nibble order) in ``layout``; ``out`` may be ``wq`` itself."""
    return _repack(wq, layout, out, to_layout=True)


def q4f16_unpack(packed: torch.Tensor, layout="paired", out: torch.Tensor | None = None) -> torch.Tensor:
    """Back to the reference's nibble order: the exact inverse of :func:`q4f16_repack`."""
    return _repack(packed, layout, out, to_layout=False)


def _repack(src: torch.Tensor, layout, out, to_layout: bool) -> torch.Tensor:
    if src.dtype not in (torch.int32, torch.uint32) or src.dim() != 2 or not src.is_contiguous():
        raise ValueError("packed weights are a contiguous 2-D 32-bit integer tensor [N, K/8]")
    if out is None:
        out = torch.empty_like(src)
    if out.shape != src.shape or out.dtype != src.dtype or out.device != src.device or not out.is_contiguous():
        raise ValueError("out must match the packed tensor")
    L = _lib.lib()
    fn = L.b200_q4f16_repack if to_layout else L.b200_q4f16_unpack
    N, K = src.shape[0], src.shape[1] * 8
    with _on(src.device):
        _lib.check(fn(src.data_ptr(), out.data_ptr(), N, K, _layout_code(layout), _stream_ptr(src.device)))
    return out


def q4f16_dequantize(wq: torch.Tensor, scales: torch.Tensor, out: torch.Tensor | None = None, layout=None) -> torch.Tensor:
    """w[N,K] fp16 = decode(wq, scales); bit-exact with the reference's decode stage."""
    if out is None:
        out = torch.empty((wq.shape[0], wq.shape[1] * 8), dtype=torch.float16, device=wq.device)
    if layout is None:
        native = _native or _torch_call()
        if native and native.dequantize(wq, scales, out):
            return out
    L = _lib.lib()
    if layout is not None:
        N, K = wq.shape[0], wq.shape[1] * 8
        with _on(wq.device):
            _lib.check(L.b200_q4f16_dequantize_layout(wq.data_ptr(), scales.data_ptr(), out.data_ptr(), N, K,
                                                      _layout_code(layout), _stream_ptr(wq.device)))
        return out
    if _dequantize_by_pointer(L, wq, scales, out):
        return out
    with _on(wq.device):
        L.b200_set_stream(_stream_ptr(wq.device))
        vw, vs, vo = (_DLView(t) for t in (wq, scales, out))
        _lib.check(L.b200_q4f16_dequantize_dl(vw.ptr(), vs.ptr(), vo.ptr()))
    return out


def launch_count() -> int:
    return int(_lib.lib().b200_launch_count())


def reset_launch_count() -> None:
    _lib.lib().b200_reset_launch_count()
