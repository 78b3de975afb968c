"""The mixed P2G's tile shapes, by the grids they are chosen for: more tiles than a wave
on thin and small ones (square tiles) and tiny batch members (half tiles), rows else.
Batches equal their members run alone bit for bit, whatever shape either takes, and
those the FP64 form: FP32 state, a few steps, 1e-5 of the field's norm."""
import time

import numpy as np
import pytest

import mpm2d

from test_gpu_step_paths import small_grid

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "vx", "vy", "v", "sxx", "sxy", "syy", "node_m", "node_vx", "node_vy")
GRIDS = {"tiny": [(2, 2), (3, 3), (5, 5), (5, 4), (3, 6)], "small": [(9, 9), (13, 13), (16, 9)],
         "thin": [(3, 301), (9, 200), (33, 130), (16, 100)], "wide": [(300, 3), (200, 33)],
         "many tiny": [(2, 2), (3, 3), (5, 5), (5, 4), (3, 6)] * 160, "many small": [(9, 9), (13, 13), (16, 9)] * 160,
         "long": [(3, 9200), (9, 6001), (33, 3001)]}


@pytest.mark.parametrize("precision", ["mixed", "mixed_f64node"])
@pytest.mark.parametrize("kind", GRIDS)
def test_shapes(kind, precision):
    members = [small_grid(nx, ny, k) for k, (nx, ny) in enumerate(GRIDS[kind])]
    batch = mpm2d.Batch(members, precision=precision)
    batch.step(5)
    for k, sc in list(enumerate(members))[-8:]:
        one = mpm2d.Simulation(sc, precision=precision)
        ref = mpm2d.Simulation(sc, precision="fp64")
        one.step(5)
        ref.step(5)
        for f in FIELDS:
            np.testing.assert_array_equal(batch.member_get(k, f), one.get(f), err_msg="%d %s" % (k, f))
        for fs in (("x", "y"), ("vx", "vy"), ("node_m",), ("node_vx", "node_vy")):
            a = np.concatenate([one.get(f) for f in fs])
            b = np.concatenate([ref.get(f) for f in fs])
            assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b), (GRIDS[kind][k], fs)


def lattice(nx, ny):
    sc = small_grid(nx, ny, 1)
    h = sc["h"]
    x, y = np.meshgrid((np.arange(2 * nx - 2) + 0.5) * h / 2, (np.arange(2 * ny - 2) + 0.5) * h / 2, indexing="ij")
    return dict(sc, particles=dict(sc["particles"], x=x.ravel(), y=y.ravel()), xmax=nx * h, ymax=ny * h, gravity=0.0)


def test_thin_grids_take_few_tiles():
    """A grid of one column of tiles steps in about the time of its transpose: at most 1.8 times
    (two thirds of the kernels' time is the particles', and the same)."""
    best = {}
    for nx, ny in ((3, 20001), (20001, 3)):
        sim = mpm2d.Simulation(lattice(nx, ny), precision="mixed")
        sim.step(16)
        sim.synchronize()
        best[nx] = np.inf
        for _ in range(5):
            start = time.perf_counter()
            sim.step(64)
            sim.synchronize()
            best[nx] = min(best[nx], time.perf_counter() - start)
        sim.close()
    assert best[3] <= 1.8 * best[20001], best
