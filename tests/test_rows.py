"""Sizes of the FP64 step's element rows (tests/cpp/rows_check.cpp, built here
with g++): the width against its rule, and a host without memory reported
instead of an exception through the C entry."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("rows") / "librows_check.so")
    src = os.path.join(ROOT, "tests", "cpp", "rows_check.cpp")
    subprocess.run([shutil.which("g++") or "g++", "-O2", "-std=c++17", "-Wl,-Bsymbolic", "-shared", "-fPIC", "-o", out,
                    src], check=True, capture_output=True)
    lib = C.CDLL(out)
    lib.row_width.argtypes = [C.POINTER(C.c_int), C.c_size_t, C.c_size_t, C.c_int, C.POINTER(C.c_int),
                              C.POINTER(C.c_size_t)]
    return lib


def width(rows, emap, ne, no_memory=0):
    e = np.ascontiguousarray(emap, dtype=np.int32)
    cap, filled = C.c_int(), C.c_size_t()
    rc = rows.row_width(e.ctypes.data_as(C.POINTER(C.c_int)), e.size, ne, no_memory, C.byref(cap), C.byref(filled))
    return rc, cap.value, filled.value


@pytest.mark.parametrize("ne", [1, 63, 64, 65, 4096])
@pytest.mark.parametrize("ppc", [0, 1, 8, 9, 33, 300])
def test_width_and_filled(rows, ne, ppc):
    rng = np.random.default_rng(ne + ppc)
    used = np.arange(ne) if ne < 4096 else np.arange(0, ne, 7)
    emap = np.repeat(used, ppc)
    rng.shuffle(emap)
    emap = np.concatenate([emap, [-1, -1, -1]])
    rc, cap, filled = width(rows, emap, ne)
    assert rc == 0 and filled == (used.size if ppc else 0)
    want = 16
    while ppc and want < 2 * ppc and (want < 64 or 2 * want * ne <= 128 * emap.size):
        want *= 2
    assert cap == want


def test_no_host_memory_is_reported(rows):
    assert width(rows, [0, 1, 1, -1], 4, no_memory=1)[0] == 1
    assert width(rows, [0, 1, 1, -1], 4) == (0, 16, 2)


@pytest.mark.parametrize("ppc", [16, 64, 1000])
def test_crowd_on_a_large_grid_takes_narrow_rows(rows, ppc):
    """Rows above 16 slots: 128 slots a particle at most, in each of two buffers."""
    ne = 1 << 22
    for crowded in (16, 4096):
        emap = np.repeat(np.arange(crowded) * 7, ppc)
        rc, cap, filled = width(rows, emap, ne)
        assert rc == 0 and filled == crowded
        assert cap == 16 or cap * ne <= 128 * emap.size


def test_sums_by_list_only_on_large_empty_grids(rows):
    rows.sums_by_list.argtypes = [C.c_size_t, C.c_size_t]
    for n, ne, want in ((0, 1, 0), (10, (1 << 24) - 1, 0), (10, 1 << 24, 1), (1 << 23, 1 << 24, 0), ((1 << 23) - 1, 1 << 24, 1),
                        (1 << 28, 1 << 29, 0), (1 << 20, 1 << 30, 1)):
        assert rows.sums_by_list(n, ne) == want, (n, ne)
