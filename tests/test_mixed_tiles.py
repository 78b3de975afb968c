"""The mixed form's tiles on long thin grids: every tile has its own row and
column, also beyond 2^16 of either (tests/cpp/tiles_check.cpp, built here with
g++), and a block near the far end of such a grid moves as the FP64 form's."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SHAPES = [(32, 8), (16, 8), (32, 16)]      # elements a tile, each variant of the kernel


@pytest.fixture(scope="module")
def tiles(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("tiles") / "libtiles_check.so")
    src = os.path.join(ROOT, "tests", "cpp", "tiles_check.cpp")
    subprocess.run([shutil.which("g++") or "g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", out, src], check=True,
                   capture_output=True)
    lib = C.CDLL(out)
    u32p = C.POINTER(C.c_uint32)
    lib.batch_tiles.argtypes, lib.batch_tiles.restype = [C.c_int, u32p, C.c_uint32, C.c_uint32, u32p], C.c_longlong
    lib.single_tiles.argtypes, lib.single_tiles.restype = [C.c_uint32, C.c_uint32, C.c_longlong, u32p], None
    return lib


def ptr(a):
    return a.ctypes.data_as(C.POINTER(C.c_uint32))


def expected(grids, width, height):
    rows = []
    for k, (Nx, Ny) in enumerate(grids):
        nx, ny = (Nx + width - 2) // (width - 1), (Ny + height - 2) // (height - 1)
        r, c = np.divmod(np.arange(nx * ny, dtype=np.int64), nx)
        rows.append(np.stack([np.full(nx * ny, k), r, c], axis=1))
    return np.concatenate(rows)


def far(width, height):
    """Grids with 65 537 tile rows, 65 537 tile columns, and the sizes around them."""
    return [(3, 65536 * (height - 1) + d) for d in (0, 1, height)] + \
           [(65536 * (width - 1) + d, 3) for d in (0, 1, width)] + [(2, 2), (65, 33)]


@pytest.mark.parametrize("width,height", SHAPES)
def test_every_tile_has_its_row_and_column(tiles, width, height):
    for Nx, Ny in far(width, height):
        want = expected([(Nx, Ny)], width, height)
        got = np.zeros((len(want), 3), dtype=np.uint32)
        tiles.single_tiles(Nx, width, len(want), ptr(got))
        assert np.array_equal(got, want), (Nx, Ny)
    grids = far(width, height)
    want = expected(grids, width, height)
    flat = np.array(grids, dtype=np.uint32).ravel()
    assert tiles.batch_tiles(len(grids), ptr(flat), width, height, None) == len(want)
    got = np.zeros((len(want), 3), dtype=np.uint32)
    tiles.batch_tiles(len(grids), ptr(flat), width, height, ptr(got))
    assert np.array_equal(got, want)


def tower(cells_y, nx, near_top):
    """A falling block of 2 x 2 particles an element, four elements high, on a
    tower of 3 x cells_y elements of side 1: at its foot or just below its top."""
    h = 1.0
    y0 = cells_y - 16 if near_top else 8
    a = (np.arange(2 * (nx - 1)) + 0.5) * 0.5
    X, Y = np.meshgrid(a, y0 + (np.arange(8) + 0.5) * 0.5, indexing="ij")
    n = X.size
    p = {"m": np.full(n, 0.25 * 1500), "v": np.full(n, 0.25), "x": X.ravel(), "y": Y.ravel(), "vx": np.zeros(n),
         "vy": np.full(n, -0.25), "sxx": np.zeros(n), "sxy": np.zeros(n), "syy": np.zeros(n)}
    return {"Nx": nx, "Ny": cells_y + 1, "h": h, "dt": 1e-2, "material": "isolin", "props": [1e3, 0.3], "bc": "box",
            "bcf": [0.0, 0.0, 1.0, 1.0], "bci": [1, 3, 1, 0], "gravity": -9.8, "particles": p,
            "xmax": (nx - 1) * h, "ymax": cells_y * h}


# 65 538 tile rows of 7 nodes
TALL = 65538 * 7


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [False, True])
def test_far_end_of_a_tall_grid_vs_fp64(batch):
    """Relative bounds of the mixed form against the FP64 form over a few steps
    (FP32 state: 2^-24 a rounding, some hundred of them a step on values of
    order one: 1e-4)."""
    import mpm2d
    steps = 5
    ref = mpm2d.Simulation(tower(TALL, 4, True))
    ref.step(steps)
    if batch:
        sim = mpm2d.Batch([tower(64, 4, False), tower(TALL, 4, True)])
    else:
        sim = mpm2d.Simulation(tower(TALL, 4, True), precision="mixed")
    sim.step(steps)
    get = (lambda k: sim.member_get(1, k)) if batch else sim.get
    dy = ref.get("y") - tower(TALL, 4, True)["particles"]["y"]
    assert dy.min() < 0 and np.all(np.abs(dy) < 0.1)
    for k in ("x", "y"):
        assert np.abs(get(k) - ref.get(k)).max() < 1e-5, k
    for k, scale in (("vx", 1.0), ("vy", 1.0)):
        assert np.abs(get(k) - ref.get(k)).max() < 1e-4 * scale, k
    m, want = get("node_m"), ref.get("node_m")
    assert np.abs(m - want).max() < 1e-4 * want.max() and np.array_equal(m > 0, want > 0)
