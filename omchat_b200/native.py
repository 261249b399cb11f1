"""How the C entries are called: by csrc/call.cpp where it could be built, else by ctypes. Either way a pointer argument may be a tensor, None or an address."""
from __future__ import annotations

import ctypes
import importlib.util
import warnings
from ctypes import c_float, c_int, c_longlong, c_void_p
from typing import Optional

import torch

_KINDS = {c_void_p: "P", c_int: "I", c_longlong: "L", c_float: "F"}


class Pointer:
    """Argument type of ctypes that takes tensors too."""

    @staticmethod
    def from_param(v):
        return c_void_p.from_param(v.data_ptr() if isinstance(v, torch.Tensor) else v)


_module, _tried, _error = None, False, RuntimeError


def module(compile: bool = True):
    """The compiled calls, or None where there are none (no compiler or headers): ctypes then, several times slower per call. One that does not compile or load is
    said, once. compile False: as far as it is built already."""
    global _module, _tried
    if _module is None and not _tried:
        _tried = compile
        try:
            from . import build
            path = build.ensure_call(compile=compile)
            if path is not None:
                spec = importlib.util.spec_from_file_location("omc_call", path)
                loaded = importlib.util.module_from_spec(spec)
                spec.loader.exec_module(loaded)
                loaded.set_error_type(_error)
                _module = loaded
        except (OSError, ImportError, RuntimeError) as e:
            _tried = True
            lines = [line.strip() for line in str(e).splitlines() if line.strip()] or [type(e).__name__]
            reason = next((line for line in lines if "error:" in line), lines[-1])
            warnings.warn(f"omchat_b200: the compiled calls could not be built or loaded, every call goes through ctypes (slower): {reason}", RuntimeWarning, stacklevel=2)
    return _module


class Entries:
    """The entries of a library by name; what has none here (symbols outside the header) comes from the library itself."""

    def __init__(self, cdll: ctypes.CDLL, signatures: dict, missing_ok: bool = False):
        self._cdll = cdll
        native = module()
        for name, (res, args) in signatures.items():
            fn = getattr(cdll, name, None) if missing_ok else getattr(cdll, name)   # AttributeError if the library does not export a declared symbol
            if fn is None:
                continue
            fn.restype = res
            fn.argtypes = [Pointer if a is c_void_p else a for a in args]
            entry = None
            if native is not None and res is c_int and all(a in _KINDS for a in args):
                entry = native.entry(ctypes.cast(fn, c_void_p).value, "".join(_KINDS[a] for a in args), fn)
            setattr(self, name, fn if entry is None else entry)

    def __getattr__(self, name):
        return getattr(self.__dict__["_cdll"], name)


def need_cuda(error: type):
    """A function of tensors (or None) that raises `error` for one that is not on the current GPU. Every kernel is launched on the current stream of the CURRENT
    device: a tensor living on another GPU would be dereferenced there (illegal access or silent peer traffic), so that is an error, not a convention."""
    global _error
    _error = error
    native = module(compile=False)            # nothing is compiled while the package is imported
    if native is not None:
        native.set_error_type(error)
        return native.need_cuda

    def check(*ts):
        if _module is not None:               # compiled meanwhile
            return _module.need_cuda(*ts)
        cur: Optional[int] = None
        for t in ts:
            if t is None:
                continue
            if not t.is_cuda:
                raise error("omchat_b200 kernels need CUDA tensors (no CPU fallback)")
            if cur is None:
                cur = torch.cuda.current_device()
            if t.device.index != cur:
                raise error(f"tensor on cuda:{t.device.index} but the current device is cuda:{cur}: run the call under "
                            f"`with torch.cuda.device({t.device.index}):` (the model classes do this themselves)")
    return check


def raw_stream() -> int:
    """The current stream of the current device."""
    return torch.cuda.current_stream().cuda_stream


if hasattr(torch._C, "_cuda_getCurrentRawStream") and hasattr(torch._C, "_cuda_getDevice"):
    def raw_stream(_stream=torch._C._cuda_getCurrentRawStream, _device=torch._C._cuda_getDevice) -> int:  # noqa: F811
        """The current stream of the current device, without the objects that torch.cuda.current_stream() makes of it."""
        return _stream(_device())
