"""The checked build's limiter that takes the node bounds itself, on the CPU: an index out of range
among those it gathers is recorded under the limiter's kernel number and the element, and the
element is left as it was; the element kernels' test of an element's three edges, at which an
element whose flux was not taken is left alone."""
from __future__ import annotations

import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
LIMITER, ELEMENTS, ELEMENT = 4, 2, 1  # the kernels' numbers; the element that the harness runs


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    path = str(tmp_path_factory.mktemp("checked") / "libchecked_host.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-w", "-x", "c++",
                    *(f"-D__{w}__=" for w in ("host", "device", "noinline", "global", "grid_constant")),
                    "-D__forceinline__=inline", "-D__shared__=static", "-D__launch_bounds__(...)=", "-o", path,
                    os.path.join(HERE, "checked_host.cpp")], check=True)
    lib = C.CDLL(path)
    lib.dgr_t_bad_index.restype = lib.dgr_t_bad_edge.restype = C.c_ulonglong
    return lib


def test_nothing_wrong(lib):
    touched = C.c_int()
    assert lib.dgr_t_bad_index(0, C.byref(touched)) == 2**64 - 1
    assert touched.value


@pytest.mark.parametrize("where", [1, 2, 3, 4, 5])
def test_bad_index_is_the_limiters(lib, where):
    touched = C.c_int()
    assert lib.dgr_t_bad_index(where, C.byref(touched)) == LIMITER << 32 | ELEMENT
    assert not touched.value


@pytest.mark.parametrize("at", [-1, 0, 1, 2])
def test_bad_edge_of_an_element(lib, at):
    ok = C.c_int()
    want = 2**64 - 1 if at < 0 else ELEMENTS << 32 | ELEMENT
    assert lib.dgr_t_bad_edge(at, C.byref(ok)) == want
    assert ok.value == (at < 0)
