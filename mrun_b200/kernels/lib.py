"""Loads the compiled kernel libraries through their C ABI.

There is no other implementation behind these calls: if a library cannot be built or opened the
import fails with the reason, and every entry point raises :class:`KernelError` with the
library's own message when it refuses its arguments.
"""
from __future__ import annotations

import ctypes
import os
import re
from typing import Dict, Optional

from . import build


class KernelError(RuntimeError):
    pass


_PROTOTYPE = re.compile(r"MRUN_API\s+(?:int|long)\s+(\w+)\(([^)]*)\)\s*\{")
_prototypes: Optional[Dict[str, list]] = None


def _parameter_type(declaration: str):
    if "*" in declaration or "cudaStream_t" in declaration:
        return ctypes.c_void_p
    for word, kind in (("double", ctypes.c_double), ("float", ctypes.c_float), ("long", ctypes.c_long), ("int", ctypes.c_int)):
        if word in declaration.split():
            return kind
    raise KernelError(f"a parameter of the C ABI has no type that Python passes: {declaration.strip()!r}")


def prototypes() -> Dict[str, list]:
    """The parameter types of every entry point, read from the definitions in the sources that the libraries are built
    from.  With them a call takes plain numbers and addresses; a ctypes object an argument took a fifth of the host time of
    an uncaptured step."""
    global _prototypes
    if _prototypes is None:
        found = {}
        for name in sorted(os.listdir(build.CSRC)):
            if name.endswith(".cu"):
                with open(os.path.join(build.CSRC, name)) as f:
                    for entry, parameters in _PROTOTYPE.findall(f.read()):
                        found[entry] = [_parameter_type(p) for p in parameters.split(",") if p.strip()]
        _prototypes = found
    return _prototypes


def _undeclared(path: str, name: str, fn):
    """A function that the sources do not define: ctypes would cut a plain number to a 32-bit int, so it takes ctypes objects only."""
    def call(*args):
        for position, value in enumerate(args):
            if isinstance(value, (int, float)):
                raise KernelError(f"{name} of {path} has no declared parameters: argument {position} must say its type "
                                  f"(a ctypes object), not {value!r}")
        return fn(*args)
    return call


class Library:
    """A loaded ``.so``: ``lib.call("mrun_x", args...)`` raises on a non-zero return."""

    def __init__(self, path: str, error_symbol: str = "mrun_last_error"):
        self.path = path
        try:
            self._dll = ctypes.CDLL(path, mode=ctypes.RTLD_LOCAL)
        except OSError as error:
            raise KernelError(f"cannot open the kernel library {path}: {error}") from None
        self._last_error = getattr(self._dll, error_symbol)
        self._last_error.restype = ctypes.c_char_p
        self._functions: Dict[str, ctypes._CFuncPtr] = {}

    def function(self, name: str):
        fn = self._functions.get(name)
        if fn is None:
            try:
                fn = getattr(self._dll, name)
            except AttributeError:
                raise KernelError(f"{self.path} exports no {name}") from None
            fn.restype = ctypes.c_int
            types = prototypes().get(name)
            if types is None:
                fn = _undeclared(self.path, name, fn)
            else:
                fn.argtypes = types
            self._functions[name] = fn
        return fn

    def call(self, name: str, *args) -> None:
        global _calls
        _calls += 1
        if (self._functions.get(name) or self.function(name))(*args) != 0:
            raise KernelError(self._last_error().decode("utf-8", "replace"))


_calls = 0


def call_count() -> int:
    """How many kernel entry points were called so far (each launches this library's kernels)."""
    return _calls


_core: Library | None = None
_attention: Dict[tuple, Library] = {}


def core() -> Library:
    global _core
    if _core is None:
        lib = Library(build.build_core())
        arch = lib._dll.mrun_target_arch
        arch.restype = ctypes.c_int
        if arch() != 100:
            raise KernelError(f"{lib.path} was not built for sm_100a")
        _core = lib
    return _core


def attention(head_dim: int, value_dim: int | None = None, scored: bool = False) -> Library:
    """The tensor-core attention library for ``head_dim`` (and another ``value_dim``, and with a score
    form), built at first use."""
    value_dim = head_dim if value_dim is None else value_dim
    key = (head_dim, value_dim, bool(scored))
    lib = _attention.get(key)
    if lib is None:
        lib = Library(build.build_attention(head_dim, value_dim, scored))
        found = tuple(int(getattr(lib._dll, f"mrun_attn_{what}")()) for what in ("head_dim", "value_dim", "scored"))
        if found != (head_dim, value_dim, int(scored)):
            raise KernelError(f"{lib.path} was built for {found}, not {(head_dim, value_dim, int(scored))}")
        _attention[key] = lib
    return lib
