"""FP64 step: rows sized for the initial positions, and particles that crowd later.

Particles at four an element are set to 64 an element (rows hold 16).  Results
against the oracle started there: 1e-10 of each field's largest value, as for one
step from a reference state.  Time a step against a simulation created there, whose
rows are wide enough: at most four times (both order the same lists; the first also
follows a chain of 48 links a thread, of about the latency of what it then sums)."""
import numpy as np
import pytest
import torch

from conftest import field_err
from oracle import oracle as O
import mpm2d
import scenes

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "vx", "vy", "v", "sxx", "sxy", "syy", "ux", "uy", "node_m", "node_mx", "node_my")
# (the reference's nodal forces after a MUSL step are its second projection's, which no step reads)
FORCES = {"usl": ("node_fx", "node_fy"), "musl": ()}


def spread_and_packed(cells, scheme="usl", seed=None):
    spread = dict(scenes.box_fill(cells=cells, ppc_1d=2, material="g_local_mu2", dt=1e-6), scheme=scheme)
    p = {k: np.array(v) for k, v in spread["particles"].items()}
    if seed is not None:
        rng = np.random.default_rng(seed)
        n = len(p["x"])
        p["vx"], p["vy"] = rng.uniform(-0.1, 0.1, (2, n))
        p["sxx"], p["syy"] = -rng.uniform(1e3, 2e3, (2, n))
        mixed = rng.permutation(n)          # neighbours far apart in the arrays
        p = {k: a[mixed] for k, a in p.items()}
        spread = dict(spread, particles=p)
    return spread, dict(spread, particles=dict(p, x=p["x"] * 0.25, y=p["y"] * 0.25))


def moved(spread, packed, **kw):
    sim = mpm2d.Simulation(spread, **kw)
    for k in ("x", "y"):
        sim.set(k, packed["particles"][k])
    return sim


@pytest.mark.parametrize("scheme", ["usl", "musl"])
def test_moved_crowd_vs_oracle(scheme):
    spread, packed = spread_and_packed(16, scheme, seed=3)
    sim = moved(spread, packed, store_transients=True)
    orc = O.Oracle(packed, nthreads=4)
    for _ in range(2):
        sim.step(1)
        orc.step(1)
        for f in FIELDS + FORCES[scheme]:
            assert field_err(sim.get(f), orc.get, f) <= 1e-10, (f, field_err(sim.get(f), orc.get, f))


@pytest.mark.parametrize("material, scheme", [("g_local_mu2", "usl"), ("dp_ri_mt", "musl"), ("g_local_mu2_ext", "usl"),
                                              ("g_nonlocal_mu2", "usl"), ("g_nonlocal_avg", "usl")])
def test_chains_and_rows_give_the_same_bits(material, scheme):
    """Every reader of the ordered lists: moved particles against particles created there."""
    spread, packed = spread_and_packed(16, scheme, seed=8)
    extra = {"material": material, "gravity": -9.8}
    a, b = moved(dict(spread, **extra), dict(packed, **extra)), mpm2d.Simulation(dict(packed, **extra))
    for _ in range(3):
        a.step(1)
        b.step(1)
        for f in ("x", "y", "vx", "vy", "v", "sxx", "sxy", "syy", "node_m", "node_vx", "node_gf"):
            np.testing.assert_array_equal(a.get(f), b.get(f), err_msg=f)
    for u, v in zip(a.get_map() + a.get_sort(), b.get_map() + b.get_sort()):
        np.testing.assert_array_equal(u, v)


def test_gradient_through_chains():
    spread, packed = spread_and_packed(16, seed=9)
    got = []
    for sim in (moved(spread, packed), mpm2d.Simulation(packed)):
        sim.adj_forward_tape(6, 4)
        gx = np.linspace(-1.0, 1.0, sim.n)
        grad = sim.adj_backward(gx, gx[::-1].copy())
        got.append([grad] + [sim.adj_state(k) for k in ("x", "y", "vx", "v", "sxx", "Tzz")])
    for u, v in zip(*got):
        np.testing.assert_array_equal(u, v)


def us_a_step(sim, steps=8):
    sim.step(steps)
    sim.synchronize()
    stream = torch.cuda.ExternalStream(sim.stream())
    best = np.inf
    for _ in range(3):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        sim.step(steps)
        b.record(stream)
        b.synchronize()
        best = min(best, a.elapsed_time(b) / steps * 1e3)
    return best


def test_moved_crowd_is_not_slow():
    spread, packed = spread_and_packed(256)
    there = us_a_step(mpm2d.Simulation(packed))
    later = us_a_step(moved(spread, packed))
    assert later <= 4 * there, (later, there)
