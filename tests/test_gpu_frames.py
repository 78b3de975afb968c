"""Frame read-back: fields written into pinned host arrays by the device equal
the single reads, at odd sizes and destinations of 8-byte alignment, with
fields the state does not hold as arrays, with more fields than one launch
takes, and where destinations overlap (the later field's values stay); and
pageable reads over several staging chunks equal them too."""
import numpy as np
import pytest
import torch

import mpm2d
import scenes

pytestmark = pytest.mark.gpu

FIELDS = ("m", "v", "x", "y", "vx", "vy", "sxx", "sxy", "syy", "ux", "uy", "state9", "state10")


def pinned(n, offset):
    return torch.full((n + offset,), -7.0, dtype=torch.float64, pin_memory=True).numpy()[offset:]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("cells,ppc,offset", [(3, 3, 0), (9, 3, 1), (300, 2, 1)])
def test_frames_equal_single_reads(precision, cells, ppc, offset):
    sc = scenes.box_fill(cells=cells, ppc_1d=ppc, material="g_local_mu2", dt=1e-5)
    sim = mpm2d.Simulation(sc, precision=precision)
    sim.step(3)
    names = FIELDS + ("Tzz", "node_m", "node_vy") + (("by", "node_ax", "v0") if precision == "fp64" else ("node_ax",))
    want = {k: sim.get(k).copy() for k in names}
    out = {k: pinned(len(want[k]), offset) for k in names}
    got = sim.get_frame(names, out=out)
    for k in names:
        assert got[k] is out[k]
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    for k, a in sim.get_frame(names).items():       # pageable
        np.testing.assert_array_equal(a, want[k], err_msg=k)
    # x over the first half of y's destination, then y: y whole, x's rest
    n = sim.n
    both = pinned(n + n // 2, offset)
    sim.get_frame(("x", "y"), out={"x": both[:n], "y": both[n // 2:]})
    np.testing.assert_array_equal(both[:n // 2], want["x"][:n // 2])
    np.testing.assert_array_equal(both[n // 2:], want["y"])
