"""third(x) of the limiter (x / 3 by a reciprocal and two corrections) equals the IEEE division
bit for bit over the whole range of doubles: subnormals, powers of two and their neighbours,
signed zeros, infinities."""
from __future__ import annotations

import ctypes as C
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_third_equals_division(tmp_path):
    lib_path = str(tmp_path / "libthird_host.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-x", "c++",
                    "-D__host__=", "-D__device__=", "-D__forceinline__=inline", "-o", lib_path,
                    os.path.join(HERE, "third_host.cpp")], check=True)
    lib = C.CDLL(lib_path)
    lib.dgr_t_third.restype = C.c_longlong
    lib.dgr_t_third.argtypes = [C.c_longlong, C.c_ulonglong]
    assert lib.dgr_t_third(4_000_000, 20250311) == 0
