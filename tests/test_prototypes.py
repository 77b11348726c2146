"""The parameter types that calls into the kernel libraries are converted with are those of the sources."""
from __future__ import annotations

import ctypes
import os
import re


def test_every_entry_point_has_its_types():
    from mrun_b200.kernels import build, lib
    text = "".join(open(os.path.join(build.CSRC, n)).read() for n in sorted(os.listdir(build.CSRC)) if n.endswith(".cu"))
    names = set(re.findall(r"MRUN_API[^(;{]*?(\w+)\(", text)) - {"mrun_last_error"}
    found = lib.prototypes()
    assert names == set(found) and len(names) > 80
    P, I, L, D = ctypes.c_void_p, ctypes.c_int, ctypes.c_long, ctypes.c_double
    assert found["mrun_rotary_table"] == [P, P, P, I, I, D, P]
    assert found["mrun_gemm_f32_nt"] == [P, P, P, I, I, I, L, L, P]
    assert found["mrun_target_arch"] == []
