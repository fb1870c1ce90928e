"""The calls of native_call.cpp through ctypes, for a machine that can compile the kernels but lacks Python's or torch's C++ headers:
the same names, `torch.mm` for the products, and no lists of launches (a prompt step of a small model then takes 10 us a launch)."""

from __future__ import annotations

import ctypes

import torch

from .launchers import F, I, LAUNCHERS, LL, P, QUERIES


class _Pointer(ctypes.c_void_p):
    """None, an address, or a tensor."""

    @classmethod
    def from_param(cls, value):
        return ctypes.c_void_p(value.data_ptr() if isinstance(value, torch.Tensor) else value)


_KINDS = {P: _Pointer, I: ctypes.c_int, F: ctypes.c_float, LL: ctypes.c_longlong, None: None}


class PlainCalls:
    def set_slow_need(self, check) -> None:
        self.need = check

    def bind(self, name: str, address: int):
        result, types = (I, LAUNCHERS[name]) if name in LAUNCHERS else QUERIES[name]
        fn = ctypes.CFUNCTYPE(_KINDS[result])(address)
        fn.argtypes = [_KINDS[t] for t in types]
        return fn

    @staticmethod
    def ptr(t):
        return None if t is None else t.data_ptr()

    @staticmethod
    def stream() -> int:
        return torch.cuda.current_stream().cuda_stream

    @staticmethod
    def mm(x, w, out) -> bool:
        return False

    def record(self) -> None:
        pass

    def unlisted(self) -> None:
        pass

    def recorded(self) -> None:
        return None
