"""Functions whose parameters' types nobody declared: what a program hands to an exported C symbol that it opened itself arrives
whole, and a library's function that the sources do not define takes no plain numbers."""
from __future__ import annotations

import ctypes
import subprocess
import sys

import pytest
import torch


def test_an_address_reaches_an_undeclared_function_whole():
    """In a process of its own: an address cut to 32 bits ends it."""
    script = """
import ctypes, torch
from mrun_b200.kernels.ops import _ptr
src, dst = torch.arange(1 << 20, dtype=torch.int32), torch.zeros(1 << 20, dtype=torch.int32)
assert src.data_ptr() >> 32
copy = ctypes.CDLL(None).memcpy
copy(_ptr(dst), _ptr(src), ctypes.c_size_t(4 << 20))
assert torch.equal(src, dst) and not _ptr(None).value
"""
    done = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, timeout=600)
    assert done.returncode == 0, done.stderr


def test_a_stream_is_a_whole_handle(monkeypatch):
    from mrun_b200.kernels import ops
    handle = 0x7f0123456789ab0
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: 0, raising=False)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: handle, raising=False)
    assert isinstance(ops._stream(), ctypes.c_void_p) and ops._stream().value == handle


def test_a_function_without_types_refuses_plain_numbers(tmp_path):
    """A number that is not declared as an address would be cut to 32 bits in silence."""
    from mrun_b200.kernels import build, lib
    source, target = tmp_path / "other.cpp", str(tmp_path / "libother.so")
    source.write_text('extern "C" { const char* mrun_last_error() { return "no"; }\n'
                      'int other(void* a) { return a != (void*)0x7f0123456789ab0; } }\n')
    subprocess.run([build.find_cxx(), "-shared", "-fPIC", "-o", target, str(source)], check=True)
    library = lib.Library(target)
    with pytest.raises(lib.KernelError, match="other"):
        library.call("other", 0x7f0123456789ab0)
    library.call("other", ctypes.c_void_p(0x7f0123456789ab0))
