"""Mixed form: elements with more particles than a tile stages are ordered in global
memory, by heap sort.  Against the FP64 form (FP32 sums of 1600 terms: 1e-4 of the
norm), and in a time that grows with the particles and not with their square: four
times the particles an element, six times the time at most."""
import time

import numpy as np
import pytest

import mpm2d
import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("members", [None, 2])
def test_long_lists_in_global_memory(members):
    seconds = {}
    for ppc in (20, 40):
        sc = scenes.box_fill(cells=8, ppc_1d=ppc)
        rng = np.random.default_rng(ppc)
        p = sc["particles"]
        p["vx"], p["vy"] = rng.uniform(-0.1, 0.1, (2, len(p["x"])))
        mixed = rng.permutation(len(p["x"]))
        sc = dict(sc, particles={k: a[mixed] for k, a in p.items()})
        sim = mpm2d.Simulation(sc, precision="mixed") if members is None else mpm2d.Batch([sc] * members)
        sim.step(1)
        sim.synchronize()
        start = time.perf_counter()
        sim.step(1)
        sim.synchronize()
        seconds[ppc] = time.perf_counter() - start
        ref = mpm2d.Simulation(sc)
        ref.step(2)
        for k in ("x", "vx", "vy", "node_m", "node_vx"):
            want = ref.get(k)
            for got in ([sim.get(k)] if members is None else [sim.member_get(m, k) for m in range(members)]):
                assert np.linalg.norm(got - want) <= 1e-4 * np.linalg.norm(want), (ppc, k)
        ref.close()
        sim.close()
    assert seconds[40] <= 6 * seconds[20], seconds
