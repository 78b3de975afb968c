"""What reads cost beside their bytes.  A field read into pageable pages that are
mapped takes the time of its bytes over the link, as into pinned memory (the device
writes both): at most four times that."""
import mmap
import time

import numpy as np
import pytest
import torch

import mpm2d
import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_pageable_reads_cost_their_bytes(precision):
    sim = mpm2d.Simulation(scenes.box_fill(cells=512, material="isolin"), precision=precision)
    sim.step(1)

    def best(array):
        t = np.inf
        for _ in range(10):
            start = time.perf_counter()
            sim.get_frame(["x"], out={"x": array})
            t = min(t, time.perf_counter() - start)
        return t

    pageable = np.zeros(sim.n)                 # the zeros are written: its pages are mapped
    pageable[:] = 1.0
    pinned = torch.zeros(sim.n, dtype=torch.float64, pin_memory=True).numpy()
    there, here = best(pinned), best(pageable)
    np.testing.assert_array_equal(pageable, pinned)
    assert here <= 4 * there, (here, there)
    sim.close()


def test_reads_into_fresh_and_partly_mapped_pages():
    sim = mpm2d.Simulation(scenes.box_fill(cells=256, material="isolin"))
    sim.step(1)
    want = sim.get("x").copy()
    for touched in ([], [0], [-1], [0, -1], [sim.n // 2]):
        a = np.empty(sim.n + 3)[3:]
        a[touched] = 5.0
        np.testing.assert_array_equal(sim.get_frame(["x"], out={"x": a})["x"], want)
    fresh = np.frombuffer(mmap.mmap(-1, 8 * sim.n + 8), dtype=np.float64)[1:]   # no page of it mapped
    np.testing.assert_array_equal(sim.get_frame(["x"], out={"x": fresh})["x"], want)
    sim.close()


def test_partly_mapped_arrays_cost_no_more_than_fresh_ones():
    """An array grown by its allocator: some pages mapped, the rest not (twice the fresh array's time at most)."""
    sim = mpm2d.Simulation(scenes.box_fill(cells=128, material="isolin"))
    sim.step(1)

    def best(touched):
        t = np.inf
        for _ in range(15):
            a = np.frombuffer(mmap.mmap(-1, 8 * sim.n), dtype=np.float64)
            a[touched] = 1.0
            start = time.perf_counter()
            sim.get_frame(["x"], out={"x": a})
            t = min(t, time.perf_counter() - start)
        return t

    best([])
    fresh = best([])
    for touched in ([0], [-1], [0, -1]):
        assert best(touched) <= 2 * fresh, (touched, best(touched), fresh)
    sim.close()


def test_a_mixed_field_is_one_launch():
    """No permutation formed for a single field, and the values of the frame export (bit for bit)."""
    for members in (None, 3):
        sc = scenes.box_fill(cells=40, material="g_local_mu2")
        sim = mpm2d.Simulation(sc, precision="mixed") if members is None else mpm2d.Batch([sc] * members)
        sim.step(3)
        sim.synchronize()
        names = ["x", "y", "vx", "syy", "v", "Tzz"]
        out = {k: torch.zeros(sim.n, dtype=torch.float64, pin_memory=True).numpy() for k in names}
        frame = sim.get_frame(names, out=out)
        for k in names:
            before = sim.launch_count()
            np.testing.assert_array_equal(sim.get(k), frame[k])
            assert sim.launch_count() - before == 1
        sim.close()
