"""Arrays that a call allocates on first need come all or none: after an
allocation that failed at any of them nothing is held and no pointer is set, and
the next call allocates them all (tests/cpp/alloc_check.cpp, built with g++)."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("alloc") / "liballoc_check.so")
    src = os.path.join(ROOT, "tests", "cpp", "alloc_check.cpp")
    subprocess.run([shutil.which("g++") or "g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", out, src], check=True,
                   capture_output=True)
    fn = C.CDLL(out).fail_then_succeed
    fn.argtypes = [C.c_int, C.POINTER(C.c_size_t), C.c_int]
    return fn


@pytest.mark.parametrize("count", [1, 2, 5])
def test_all_or_none(check, count):
    sizes = (C.c_size_t * 16)(*[0 if k == 1 else 8 << k for k in range(16)])
    for fail_at in range(count):
        assert check(count, sizes, fail_at) == 0, fail_at
