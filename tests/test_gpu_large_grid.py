"""FP64 form on a large empty grid: sums and coefficients for the filled elements alone.

The particles lie in the lowest rows of a 4097 x 4097 grid, and of a 4097 x 65 one, whose
sums are kept by element: the same particles, elements and nodes, the same bits."""
import numpy as np
import pytest
import torch

import mpm2d
import scenes

pytestmark = pytest.mark.gpu

N = 4097


def low(Ny, material, scheme):
    h = 1.0 / (N - 1)
    rng = np.random.default_rng(11)
    sc = scenes.with_particles(scenes.box_fill(cells=64, material=material), np.arange(6000))
    p = dict(sc["particles"])
    n = len(p["x"])
    p["x"], p["y"] = rng.uniform(0.0, 1.0, n), rng.uniform(0.0, 30 * h, n)
    p["x"][:900] = 0.5 + rng.uniform(0, 3 * h, 900)        # crowded elements, beyond their rows
    p["y"][:900] = rng.uniform(0, 2 * h, 900)
    p["v"], p["m"] = np.full(n, h * h / 4), np.full(n, 2450.0 * h * h / 4)
    p["vx"], p["vy"] = rng.uniform(-0.1, 0.1, (2, n))
    p["syy"] = -rng.uniform(1e3, 2e3, n)
    return dict(sc, Nx=N, Ny=Ny, h=h, xmax=1.0, ymax=(Ny - 1) * h, dt=1e-7, gravity=-9.8, scheme=scheme, particles=p)


@pytest.mark.parametrize("material, scheme", [("g_local_mu2", "usl"), ("isolin", "musl"), ("g_local_mu2_ext", "usl")])
def test_large_and_small_grid_agree(material, scheme):
    large, small = (mpm2d.Simulation(low(Ny, material, scheme)) for Ny in (N, 65))
    for steps in (1, 9):
        large.step(steps)
        small.step(steps)
        for f in ("x", "y", "vx", "vy", "v", "sxx", "sxy", "syy"):
            np.testing.assert_array_equal(large.get(f), small.get(f), err_msg=f)
        for f in ("node_m", "node_vx", "node_ay"):
            a, b = large.get(f), small.get(f)
            np.testing.assert_array_equal(a[:N * 64], b[:N * 64], err_msg=f)
            assert not a[N * 64:].any()
    np.testing.assert_array_equal(large.get_map()[0], small.get_map()[0])
    large.close()
    small.close()


def test_memory_of_an_empty_element():
    torch.cuda.init()

    def used(cells):
        sc = scenes.with_particles(scenes.box_fill(cells=64, material="isolin"), np.arange(100))
        sc = dict(sc, Nx=cells + 1, Ny=cells + 1, h=1.0 / cells)
        before = torch.cuda.mem_get_info()[0]
        sim = mpm2d.Simulation(sc)
        sim.step(1)
        sim.synchronize()
        after = torch.cuda.mem_get_info()[0]
        sim.close()
        return before - after

    used(64)
    # 220 bytes an element before the rows; some megabytes for what is not the grid's
    assert used(5000) <= 220 * 5000 ** 2 + (64 << 20)
