"""CPU tests of what the library does when the CUDA runtime refuses a launch, an allocation or a
copy: its object files linked with a runtime that can be made to (fake_cuda.cpp)."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from treecorr_gb300 import build as tb
    tb.build()
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    out = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    objs = [os.path.join(tb.OUT, s.replace(".cu", ".o")) for s in tb.SOURCES]
    # (-Bsymbolic: its own CUDA calls, whatever runtime the process has loaded)
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-std=c++17", "-I", os.path.join(cuda, "include"),
                    os.path.join(HERE, "fake_cuda.cpp"), *objs, "-o", out, "-Wl,-Bsymbolic", "-pthread"],
                   check=True)
    L = ctypes.CDLL(out)
    for f in ("launches", "allocs", "bytes", "streams"):
        getattr(L, "fake_" + f).restype = ctypes.c_longlong
    for f in ("fail_launch", "fail_allocs_from"):
        getattr(L, "fake_" + f).argtypes = [ctypes.c_longlong]
        getattr(L, "fake_" + f).restype = None
    L.fake_word.restype = ctypes.POINTER(ctypes.c_int)
    L.tc_last_error.restype = ctypes.c_char_p
    L.tc_field_ntop.restype = ctypes.c_int64
    L.tc_field_ntop.argtypes = [ctypes.c_void_p]
    L.tc_field_free.argtypes = [ctypes.c_void_p]
    L.fake_reset()
    L.path = out
    return L


def _create(L, n):
    x = np.arange(n, dtype=float)
    w = np.ones(n)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    h = ctypes.c_void_p()
    d = ctypes.c_double
    rc = L.tc_field_create(0, 1, p(x), p(x), None, None, None, p(w), None, ctypes.c_int64(n), d(0.), d(1.),
                           2, ctypes.c_int64(0), 0, 3, 10, ctypes.byref(h))
    return rc, h


@pytest.mark.parametrize("n", [200, 3000])
def test_create_reports_every_launch(lib, n):
    lib.fake_reset()
    rc, h = _create(lib, n)
    assert rc == 0
    lib.tc_field_free(h)
    count, before = lib.fake_launches(), lib.fake_bytes()
    for k in range(count):
        lib.fake_reset()
        lib.fake_fail_launch(k)
        rc, h = _create(lib, n)
        assert rc != 0 and not h.value, k
        assert lib.fake_bytes() == before
    lib.fake_reset()


def test_build_reports_its_first_launch(lib):
    """(The launch that sets up the first level; without it the others work on unwritten tasks.)"""
    lib.fake_reset()
    rc, h = _create(lib, 3000)
    at = lib.fake_launches()
    lib.fake_fail_launch(at)
    assert lib.tc_field_ntop(h) < 0
    assert lib.fake_launches() == at + 1, "launches after the one that failed"
    lib.tc_field_free(h)
    lib.fake_reset()


def test_one_stream_for_all_threads(lib):
    """Allocations and kernels are ordered by the library's one stream: first calls from several
    threads must not each make one.  (A process of its own: the first call comes once.)"""
    code = """
import ctypes, sys, threading
L = ctypes.CDLL(sys.argv[1])
L.fake_streams.restype = ctypes.c_longlong
L.fake_slow_streams(200)
go = threading.Barrier(8)
def call():
    go.wait()
    L.tc_trim_memory()
t = [threading.Thread(target=call) for _ in range(8)]
[x.start() for x in t]
[x.join() for x in t]
print(L.fake_streams())
"""
    r = subprocess.run([sys.executable, "-c", code, lib.path], capture_output=True, text=True, check=True)
    assert r.stdout.split() == ["1"]
