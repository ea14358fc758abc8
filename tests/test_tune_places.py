"""Where the K1 autotuner's launches keep their four histories: places of their own, so that a sample
moves the memory that a step moves."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "afid-murphfi_b200", "csrc")


@pytest.fixture(scope="module")
def places(tmp_path_factory):
    d = tmp_path_factory.mktemp("tune")
    (d / "t.cpp").write_text('#include "afid_tune.h"\n'
                             'extern "C" size_t places(size_t bytes, size_t d0, size_t d1, int *mem, size_t *off) {\n'
                             '  const size_t dead[2] = {d0, d1};\n  afid::TunePlace p[4];\n'
                             '  const size_t need = afid::tune_places(bytes, dead, p);\n'
                             '  for (int q = 0; q < 4; ++q) { mem[q] = p[q].mem; off[q] = p[q].offset; }\n'
                             '  return need;\n}\n')
    so = str(d / "t.so")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", so, str(d / "t.cpp")], check=True)
    lib = ctypes.CDLL(so)
    lib.places.restype = ctypes.c_size_t
    lib.places.argtypes = [ctypes.c_size_t] * 3 + [ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_size_t)]
    return lib.places


@pytest.mark.parametrize("bytes_,dead", [(100, (400, 0)), (100, (399, 100)), (100, (250, 250)), (100, (100, 97)),
                                         (100, (99, 99)), (100, (150, 200)), (1, (0, 3))])
def test_places_are_disjoint_and_inside(places, bytes_, dead):
    mem, off = (ctypes.c_int * 4)(), (ctypes.c_size_t * 4)()
    need = places(bytes_, *dead, mem, off)
    size = (dead[0], dead[1], need)
    got = sorted((mem[q], off[q]) for q in range(4))
    for (m0, a), (m1, b) in zip(got, got[1:]):
        assert m0 != m1 or b - a >= bytes_
    assert all(o + bytes_ <= size[m] for m, o in got)
    # scratch only for what the dead memory does not hold
    assert need == bytes_ * max(0, 4 - dead[0] // bytes_ - dead[1] // bytes_)
