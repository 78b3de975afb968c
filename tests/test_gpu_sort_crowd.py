"""mpmg_get_sort of the FP64 form: the stable sort of the element map, in a time that
does not depend on how the particles crowd (900 an element against 4: three times at
most; the arrays read back are nearly the same)."""
import time

import numpy as np
import pytest

import mpm2d
import scenes

pytestmark = pytest.mark.gpu


def test_sort_of_a_crowd():
    best = {}
    for cells, ppc in ((256, 2), (16, 30)):
        sc = scenes.box_fill(cells=cells, ppc_1d=ppc, material="isolin")
        mixed = np.random.default_rng(5).permutation(len(sc["particles"]["x"]))
        p = {k: a[mixed] for k, a in sc["particles"].items()}
        p["x"][::97] += 1.0                     # outside the grid
        sim = mpm2d.Simulation(dict(sc, particles=p))
        sim.step(2)
        elem, active = sim.get_map()
        key = np.where(active != 0, elem, sim.ne)
        t = np.inf
        for _ in range(5):
            start = time.perf_counter()
            keys, perm, first = sim.get_sort()
            t = min(t, time.perf_counter() - start)
        best[ppc] = t
        want = np.argsort(key, kind="stable")
        assert np.array_equal(perm, want) and np.array_equal(keys, key[want])
        assert np.array_equal(first, np.searchsorted(keys, np.arange(sim.ne + 1)))
        sim.close()
    assert best[30] <= 3 * best[2], best
