"""The memory that the standalone entry points keep between calls gives way to
allocations that would not fit beside it: a larger standalone call's, a job's,
another thread's.  The library's workspace runs over an allocator of fixed size
(tests/harness/workspace.cpp)."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MB = 1 << 20


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++")
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    if not cxx or not os.path.exists(os.path.join(cuda_inc, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers are missing")
    out = str(tmp_path_factory.mktemp("workspace") / "libworkspace.so")
    subprocess.check_call([cxx, "-O1", "-std=c++17", "-shared", "-fPIC", "-pthread", "-Wl,-Bsymbolic",
                           "-I", os.path.join(ROOT, "part_conc_spt_abc_gb300", "csrc"), "-I", cuda_inc,
                           os.path.join(ROOT, "tests", "harness", "workspace.cpp"), "-o", out])
    lib = C.CDLL(out)
    for name, args, res in (("ws_open", [C.c_size_t], C.c_void_p), ("ws_close", [C.c_void_p], C.c_size_t),
                            ("ws_used", [], C.c_size_t), ("ws_keep", [], C.c_size_t),
                            ("ws_call", [C.c_void_p, C.c_size_t, C.c_size_t], C.c_int),
                            ("ws_job", [C.c_void_p, C.c_size_t], C.c_int)):
        getattr(lib, name).argtypes, getattr(lib, name).restype = args, res
    return lib


def test_calls_keep_their_memory(lib):
    w = lib.ws_open(200 * MB)
    assert lib.ws_call(w, 3 * MB, 0) == 1 and lib.ws_used() == 4 * MB
    assert lib.ws_call(w, 2 * MB, 0) == 1 and lib.ws_used() == 4 * MB
    assert lib.ws_call(w, lib.ws_keep(), 0) == 1 and lib.ws_used() == lib.ws_keep()
    assert lib.ws_call(w, lib.ws_keep() + 1, 0) == 1 and lib.ws_used() == lib.ws_keep()
    assert lib.ws_close(w) == 0


@pytest.mark.parametrize("limit", [100 * MB, 65 * MB])
def test_larger_call_than_fits_beside_it(lib, limit):
    w = lib.ws_open(limit)
    assert lib.ws_call(w, 60 * MB, 0) == 1
    assert lib.ws_call(w, limit, 0) == 1
    assert lib.ws_call(w, limit + 1, 0) == 0
    assert lib.ws_call(w, 5 * MB, 0) == 1
    assert lib.ws_close(w) == 0


def test_job_that_does_not_fit_beside_it(lib):
    w = lib.ws_open(100 * MB)
    assert lib.ws_call(w, 60 * MB, 0) == 1
    assert lib.ws_job(w, 100 * MB) == 1 and lib.ws_used() == 0
    assert lib.ws_job(w, 100 * MB + 1) == 0
    assert lib.ws_close(w) == 0


def test_block_that_only_fits_unrounded(lib):
    w = lib.ws_open(40 * MB)
    assert lib.ws_call(w, 33 * MB, 0) == 1 and lib.ws_used() == 0  # 64 MB to keep do not fit
    assert lib.ws_call(w, 20 * MB, 0) == 1 and lib.ws_used() == 32 * MB
    assert lib.ws_call(w, 34 * MB, 0) == 1
    assert lib.ws_close(w) == 0


def test_another_threads_call(lib):
    w = lib.ws_open(100 * MB)
    assert lib.ws_call(w, 60 * MB, 30 * MB) == 1 and lib.ws_used() == 64 * MB
    assert lib.ws_call(w, 60 * MB, 50 * MB) == 0  # the first call's memory is in use
    assert lib.ws_call(w, 90 * MB, 10 * MB) == 1
    assert lib.ws_call(w, 90 * MB, 11 * MB) == 0
    assert lib.ws_close(w) == 0
