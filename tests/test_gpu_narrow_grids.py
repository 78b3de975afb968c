"""FP64 step on grids of a few columns (tiles of 8 x 16 nodes) and just beyond, against
the oracle: 1e-10 of each field's largest value, as for one step from a reference state.
And in about the time of the transposed grid: at most 1.8 times."""
import time

import numpy as np
import pytest

from conftest import field_err
from oracle import oracle as O
import mpm2d

from test_gpu_mixed_shapes import lattice
from test_gpu_step_paths import FIELDS, small_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", ["usl", "musl"])
@pytest.mark.parametrize("Nx, Ny", [(2, 2), (3, 15), (3, 16), (7, 17), (8, 31), (8, 200), (9, 46)])
def test_narrow_grids_vs_oracle(Nx, Ny, scheme):
    sc = dict(small_grid(Nx, Ny, Nx + Ny), scheme=scheme)
    sim = mpm2d.Simulation(sc, store_transients=True)
    orc = O.Oracle(sc, nthreads=2)
    for _ in range(3):
        sim.step(1)
        orc.step(1)
        np.testing.assert_array_equal(sim.get_map()[0], orc.get_map()[0])
        for f in FIELDS + ("node_m", "node_mx", "node_my"):
            assert field_err(sim.get(f), orc.get, f) <= 1e-10, (f, field_err(sim.get(f), orc.get, f))


def test_a_column_steps_like_a_row():
    best = {}
    for nx, ny in ((3, 20001), (20001, 3)):
        sim = mpm2d.Simulation(lattice(nx, ny))
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
