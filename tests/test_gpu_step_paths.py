"""The step's kernels at the edges of their dispatch and of their tiles.

FP64: elements with more particles than the staged row (16), than a row (64) and
than neither; particle counts either side of the G2P's block sizes and integer
products (2 and 16 warps a sub-partition) and filled-element counts either side
of the P2G's two forms, against the oracle.  Criterion as for one step from a
reference state: 1e-10 of each field's largest value.

Mixed: grids of one to a few elements either side of the P2G's tiles, as
batch members and alone, against the FP64 form; and tiles that particles leave.
Criterion: FP32 state, a few steps: 1e-5 of the field's norm.

Nonlocal: grids either side of the size that block 0 of the solve holds whole,
against the oracle, 1e-9 (solves to 1e-12).

Adjoint: nine particles an element (a node sums more than the first four of each
element) against central differences, 1e-3."""
import numpy as np
import pytest
import torch

from conftest import field_err, rel_err
from oracle import oracle as O
import mpm2d
import scenes

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "vx", "vy", "v", "sxx", "sxy", "syy", "ux", "uy")


def sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


def stirred(sc, seed=1):
    """The scene's particles with velocities, stresses and scattered positions."""
    rng = np.random.default_rng(seed)
    p = {k: np.array(v) for k, v in sc["particles"].items()}
    n = len(p["x"])
    for k in ("x", "y"):
        p[k] = np.clip(p[k] + rng.uniform(-0.2, 0.2, n) * sc["h"], 1e-9, None)
    p["vx"], p["vy"] = rng.uniform(-0.1, 0.1, (2, n))
    p["sxx"], p["syy"] = -rng.uniform(1e3, 2e3, (2, n))
    p["sxy"] = rng.uniform(-100, 100, n)
    return dict(sc, particles=p)


def crowded():
    """A few elements with 17, 65 and 100 particles among ordinary ones."""
    sc = scenes.box_fill(cells=9, ppc_1d=2, material="g_local_mu2", dt=1e-6)
    rng = np.random.default_rng(4)
    p = sc["particles"]
    more = {k: [] for k in p}
    for (i, j), n in {(1, 1): 17, (4, 2): 65, (7, 7): 100, (8, 0): 64}.items():
        for k in p:
            more[k].append(np.full(n, p[k][0]))
        more["x"][-1] = (i + rng.uniform(0, 1, n)) * sc["h"]
        more["y"][-1] = (j + rng.uniform(0, 1, n)) * sc["h"]
    return dict(sc, particles={k: np.concatenate([p[k]] + more[k]) for k in p})


def first(cells, ppc, n, material="isolin"):
    sc = scenes.box_fill(cells=cells, ppc_1d=ppc, material=material, dt=1e-6)
    return scenes.with_particles(sc, np.arange(n))


@pytest.mark.parametrize("case", ["crowded", "one warp a block", "two", "two, last", "four", "split P2G", "whole P2G"])
def test_fp64_step_paths_vs_oracle(case):
    w = sms() * 4 * 32                     # one warp of particles a sub-partition
    sc = {"crowded": crowded, "one warp a block": lambda: first(128, 2, 2 * w),
          "two": lambda: first(128, 2, 2 * w + 1, "g_local_mu2"), "two, last": lambda: first(300, 2, 16 * w, "g_local_mu2"),
          "four": lambda: first(300, 2, 16 * w + 1), "split P2G": lambda: first(128, 1, sms() * 64),
          "whole P2G": lambda: first(128, 1, sms() * 64 + 1)}[case]()
    sc = stirred(sc)
    sim = mpm2d.Simulation(sc, store_transients=True)
    orc = O.Oracle(sc, nthreads=4)
    for _ in range(2):
        sim.step(1)
        orc.step(1)
        np.testing.assert_array_equal(sim.get_map()[0], orc.get_map()[0])
        for f in FIELDS + ("node_m", "node_mx", "node_my", "node_fx", "node_fy"):
            assert field_err(sim.get(f), orc.get, f) <= 1e-10, (f, field_err(sim.get(f), orc.get, f))


@pytest.mark.parametrize("ppc, crowds", [(2, (127, 128, 129)), (2, (256, 257, 1025)), (12, ()), (8, (900,))])
def test_long_element_lists_vs_oracle(ppc, crowds):
    """Elements whose lists whole warps order: up to 128 particles and beyond, in rows and past them."""
    sc = scenes.box_fill(cells=9, ppc_1d=ppc, material="g_local_mu2", dt=1e-6)
    rng = np.random.default_rng(6)
    p = sc["particles"]
    more = {k: [np.full(n, p[k][0]) for n in crowds] for k in p}
    more["x"] = [(2 * j + rng.uniform(0, 1, n)) * sc["h"] for j, n in enumerate(crowds)]
    more["y"] = [(3 + j + rng.uniform(0, 1, n)) * sc["h"] for j, n in enumerate(crowds)]
    p = {k: np.concatenate([p[k]] + more[k]) for k in p}
    mixed = rng.permutation(p["x"].size)
    sc = stirred(dict(sc, particles={k: a[mixed] for k, a in p.items()}))
    sim = mpm2d.Simulation(sc, store_transients=True)
    orc = O.Oracle(sc, nthreads=4)
    for _ in range(2):
        sim.step(1)
        orc.step(1)
        np.testing.assert_array_equal(sim.get_map()[0], orc.get_map()[0])
        for f in FIELDS + ("node_m", "node_mx", "node_my", "node_fx", "node_fy"):
            assert field_err(sim.get(f), orc.get, f) <= 1e-10, (f, field_err(sim.get(f), orc.get, f))


def small_grid(nx, ny, seed):
    h = 1.0 / 64
    n = 4 * (nx - 1) * (ny - 1)
    rng = np.random.default_rng(seed)
    p = {"m": np.full(n, 2450.0 * h * h / 4), "v": np.full(n, h * h / 4), "x": rng.uniform(0, (nx - 1) * h, n),
         "y": rng.uniform(0, (ny - 1) * h, n)}
    p.update({k: np.zeros(n) for k in ("vx", "vy", "sxx", "sxy", "syy")})
    return stirred({"Nx": nx, "Ny": ny, "h": h, "dt": 1e-6, "material": "g_local_mu2", "props": [1e6, 0.3], "bc": "box",
                    "bcf": [0.0, 0.0, 1.0, 1.0], "bci": [1, 3, 1, 0], "gravity": -9.8, "particles": p}, seed)


@pytest.mark.parametrize("precision", ["mixed", "mixed_f64node"])
def test_mixed_tiles_vs_fp64(precision):
    grids = [(2, 2), (16, 17), (17, 16), (15, 31), (31, 32), (47, 3), (32, 8), (33, 7)]
    members = [small_grid(nx, ny, k) for k, (nx, ny) in enumerate(grids)]
    batch = mpm2d.Batch(members, precision=precision)
    batch.step(5)
    for k, sc in enumerate(members):
        one = mpm2d.Simulation(sc, precision=precision)
        ref = mpm2d.Simulation(sc, precision="fp64")
        one.step(5)
        ref.step(5)
        for f in FIELDS + ("node_m", "node_vx", "node_vy"):
            np.testing.assert_array_equal(batch.member_get(k, f), one.get(f), err_msg="%d %s" % (k, f))
        for fs in (("x", "y"), ("vx", "vy"), ("node_m",), ("node_vx", "node_vy")):
            a = np.concatenate([one.get(f) for f in fs])
            b = np.concatenate([ref.get(f) for f in fs])
            assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b), (grids[k], fs)


@pytest.mark.parametrize("precision", ["mixed", "mixed_f64node"])
def test_nodes_of_left_tiles_are_zero(precision):
    """A clump that crosses several tiles a step (without stiffness: the step is far
    beyond the stable one of a solid) leaves zero nodes behind."""
    sc = scenes.box_fill(cells=64, ppc_1d=2, material="isolin", dt=0.3 / 64 * 16, props=(1e-6, 0.3))
    sc = scenes.with_particles(sc, np.arange(0, 32))
    n = len(sc["particles"]["x"])
    p = dict(sc["particles"], x=np.linspace(0.02, 0.03, n), y=np.linspace(0.02, 0.03, n), vx=np.full(n, 3.0),
             vy=np.full(n, 2.0))
    sc = dict(sc, particles=p, gravity=0.0, bci=[0, 0, 0, 0])
    sim = mpm2d.Simulation(sc, precision=precision)
    for _ in range(4):
        x, y = sim.get("x"), sim.get("y")
        sim.step(1)
        m = sim.get("node_m").reshape(65, 65)
        assert abs(m.sum() - p["m"].sum()) <= 1e-6 * p["m"].sum()
        jj, ii = np.nonzero(m)
        assert ii.min() / 64 >= x.min() - 1.01 / 64 and ii.max() / 64 <= x.max() + 1.01 / 64
        assert jj.min() / 64 >= y.min() - 1.01 / 64 and jj.max() / 64 <= y.max() + 1.01 / 64
        speed = np.hypot(sim.get("node_vx"), sim.get("node_vy"))
        assert np.all((speed > 0).reshape(65, 65) <= (m > 0))


@pytest.mark.parametrize("cells", [44, 45, 64])
def test_solve_sizes_vs_oracle(cells):
    sc = scenes.silo_prestressed(cells=cells, dt=1e-5)
    sim = mpm2d.Simulation(sc, store_transients=True, solver_tol=1e-12, solver_maxit=50000)
    orc = O.Oracle(sc, nthreads=4, solver="cg", cg_tol=1e-12)
    sim.step(1)
    orc.step(1)
    rc, _, resid = sim.last_solve()
    assert rc == 0 and resid <= 1e-12
    assert rel_err(sim.get("node_gf"), orc.get("node_gf")) <= 1e-9


def test_adjoint_of_full_elements():
    theta0 = np.array([0.3819, 0.6435, 0.278, 1e6])

    def run(theta, tape=None):
        sc = scenes.column(Nx=17, Ny=17, h=1 / 16, width=0.25, height=0.4, ppc_1d=3, material="g_local_mu2", rho=2450.0,
                           props=(theta[3], 0.3), dt=1e-4, jitter=1e-3, seed=5,
                           mp={"grains_d": 5.3e-4, "mu_s": theta[0], "mu_2": theta[1], "I0": theta[2]})
        sc["gravity"] = -9.81
        sim = mpm2d.Simulation(sc)
        if tape:
            sim.adj_forward_tape(120, tape)
        else:
            sim.step(120)
        return sim

    target = run(theta0 * [1.05, 0.95, 1.0, 1.1])
    tx, ty = target.get("x"), target.get("y")
    loss = lambda s: float(np.sum((s.get("x") - tx) ** 2 + (s.get("y") - ty) ** 2))
    sim = run(theta0, tape=50)
    g = sim.adj_backward(2 * (sim.get("x") - tx), 2 * (sim.get("y") - ty))
    for k in range(4):
        step = np.zeros(4)
        step[k] = 1e-4 * theta0[k]
        fd = (loss(run(theta0 + step)) - loss(run(theta0 - step))) / (2 * step[k])
        assert abs(g[k] - fd) <= 1e-3 * abs(fd), (k, g[k], fd)
