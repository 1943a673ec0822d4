"""The j-side buffer of the symmetric pair passes holds every value that a pass
stores: value v of trial row t lies at v stride + t with the stride of the
allocation, also where a pass with more values per row (adjoint 10, MHD force
12) follows one with fewer (force 7), or the lists have become shorter."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "phantom_gb300", "csrc")


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("jbuf")
    src, so = d / "jbuf.cpp", d / "jbuf.so"
    src.write_text('#include "ph_jbuf.h"\n'
                   'extern "C" int plan(int64_t *s, int64_t *n, int64_t rows, int nj) {\n'
                   '  const auto p = ph::jbuf_plan(*s, *n, rows, nj); *s = p.stride; *n = p.doubles;\n'
                   '  return p.keep ? 1 : 0; }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, str(src), "-o", str(so)], check=True)
    L = C.CDLL(str(so))
    L.plan.argtypes = [C.POINTER(C.c_int64), C.POINTER(C.c_int64), C.c_int64, C.c_int]
    return L.plan


@pytest.mark.parametrize("calls", [
    [(100, 7), (100, 10)], [(3500, 7), (3500, 10)], [(5700, 7), (5700, 10)], [(6000, 7), (6000, 10), (6000, 3)],
    [(100000, 7), (80000, 10)], [(100000, 7), (87000, 10), (30000, 12)], [(1000, 12), (1200, 7), (900, 12)],
    [(200, 10), (90000, 7), (90000, 10), (100, 10)], [(0, 7), (40, 7), (0, 12), (40, 12)]])
def test_every_stored_value_fits(plan, calls):
    stride, doubles = C.c_int64(0), C.c_int64(0)
    for rows, nj in calls:
        plan(C.byref(stride), C.byref(doubles), rows, nj)
        assert rows <= stride.value or rows == 0
        assert rows == 0 or (nj - 1) * stride.value + rows <= doubles.value, (rows, nj)
        held = (stride.value, doubles.value)
        assert plan(C.byref(stride), C.byref(doubles), rows, nj) == 1 and held == (stride.value, doubles.value)
