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
    for f in ("launches", "allocs", "bytes", "streams", "lowered"):
        getattr(L, "fake_" + f).restype = ctypes.c_longlong
    for f in ("fail_launch", "fail_allocs_from"):
        getattr(L, "fake_" + f).argtypes = [ctypes.c_longlong]
        getattr(L, "fake_" + f).restype = None
    L.fake_word.restype = ctypes.POINTER(ctypes.c_int)
    L.tc_last_error.restype = ctypes.c_char_p
    L.tc_field_ntop.restype = ctypes.c_int64
    L.tc_field_ntop.argtypes = [ctypes.c_void_p]
    L.tc_field_free.argtypes = L.tc_corr2_free.argtypes = [ctypes.c_void_p]
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


def _corr(L, nb, slop):
    o = [np.zeros(nb) for _ in range(8)]
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    d, big = ctypes.c_double, sys.float_info.max
    c = ctypes.c_void_p()
    assert L.tc_corr2_create(0, 0, 0, d(1.), d(10.), nb, d(np.log(10.) / nb), d(slop), d(slop), d(-big), d(big),
                             d(0.), d(0.), d(0.), *map(p, o), ctypes.byref(c)) == 0
    c.outputs = o
    return c


def _patches(L, *fields):
    nb, n = 3, len(fields)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    c = _corr(L, nb, 0.1)
    i, j, res, got = np.zeros(3, np.int32), np.zeros(3, np.int32), np.zeros((3, 8, nb)), ctypes.c_int(0)
    rc = L.tc_corr2_process_patches(c, (ctypes.c_void_p * n)(*fields), n, 1, 0, 3, p(i), p(j), p(res),
                                    ctypes.byref(got))
    L.tc_corr2_free(c)
    return rc


# fields built alone and side by side (as patches)
BUILDS = {1: lambda L, f: L.tc_field_ntop(f[0]) < 0, 2: lambda L, f: _patches(L, *f) != 0}


@pytest.mark.parametrize("n", [200, 3000])
@pytest.mark.parametrize("fields", [1, 2])
def test_build_without_memory_keeps_nothing_and_can_be_repeated(lib, fields, n):
    lib.fake_reset()
    f = [_create(lib, n)[1] for _ in range(fields)]
    before, at = lib.fake_bytes(), lib.fake_allocs()
    assert lib.tc_field_ntop(_create(lib, n)[1]) >= 0
    most = lib.fake_allocs() - at                    # (of a field's creation and its build)
    for k in range(most):
        lib.fake_reset()
        lib.fake_fail_allocs_from(k)
        other = lib.fake_bytes()
        if fields == 1 and lib.tc_field_ntop(f[0]) >= 0:
            assert k > 8                             # (enough for a build)
            break
        if fields == 2:
            assert k > 16 or BUILDS[2](lib, f)
        assert lib.fake_bytes() == other, k
    lib.fake_reset()
    for h in f:
        assert lib.tc_field_ntop(h) >= 0             # (there was memory again)
        lib.tc_field_free(h)


@pytest.mark.parametrize("n", [200, 3000])
@pytest.mark.parametrize("fields", [1, 2])
def test_build_that_failed_keeps_nothing_and_is_not_repeated(lib, fields, n):
    """A build that stopped on its way has moved the points: another on them would not be this
    catalog's tree."""
    lib.fake_reset()
    h = _create(lib, n)[1]
    at = lib.fake_launches()
    assert lib.tc_field_ntop(h) >= 0
    launches = lib.fake_launches() - at              # of a build
    lib.tc_field_free(h)
    for k in range(launches):
        lib.fake_reset()
        f = [_create(lib, n)[1] for _ in range(fields)]
        before = lib.fake_bytes()
        lib.fake_fail_launch(lib.fake_launches() + k)
        assert BUILDS[fields](lib, f), k
        assert lib.fake_bytes() <= before, k
        why = lib.tc_last_error()
        lib.fake_reset()
        for q in f:
            assert lib.tc_field_ntop(q) < 0 and lib.tc_last_error() == why
            lib.tc_field_free(q)
    # an error that the kernels report: of the two fields of a group the one it is for
    lib.fake_reset()
    f = [_create(lib, n)[1]]
    word = lib.fake_word()                           # (the field's error word is the first cleared)
    before = lib.fake_bytes()
    f += [_create(lib, n)[1] for _ in range(fields - 1)]
    one = lib.fake_bytes() - before
    word[0] = 5
    assert BUILDS[fields](lib, f) and b"device error" in lib.tc_last_error()
    why = lib.tc_last_error()
    lib.fake_reset()
    for q in f[1:]:
        assert lib.tc_field_ntop(q) >= 0
        lib.tc_field_free(q)
    assert lib.fake_bytes() <= before
    assert lib.tc_field_ntop(f[0]) < 0 and lib.tc_last_error() == why
    lib.tc_field_free(f[0])


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


def test_assign_that_failed_leaves_the_callers_array(lib):
    """KMeansAssign fills an array that may have no pages yet; without a result it stays as it was."""
    lib.fake_reset()
    n, k = 200, 3
    h = _create(lib, n)[1]
    lib.fake_answer(ctypes.c_longlong(0), 1)         # (the first of a small build's: its top-level cells)
    assert lib.tc_field_ntop(h) == 1
    cen, out = np.arange(2. * k), np.arange(n, dtype=np.int64) + 7
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    lib.fake_fail_copy_to(p(out))
    rc = lib.tc_kmeans_assign(h, p(cen), k, p(out), ctypes.c_int64(n))
    assert rc != 0
    np.testing.assert_array_equal(out, np.arange(n) + 7)
    lib.fake_reset()
    lib.tc_field_free(h)


def test_shared_memory_is_only_raised(lib):
    """The dynamic shared memory that a kernel may be launched with belongs to the kernel: a call with
    fewer bins must not lower it under another thread's launch."""
    lib.fake_reset()
    h = _create(lib, 300)[1]
    before = lib.fake_lowered()
    for nb in (200, 20):
        c = _corr(lib, nb, 0.)                       # the accurate mode
        assert lib.tc_corr2_process_auto(c, h, 0, 0, 1) == 0, lib.tc_last_error()
        lib.tc_corr2_free(c)
    assert lib.fake_lowered() == before
    lib.tc_field_free(h)
