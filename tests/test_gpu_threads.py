"""Reads of one context from several host threads: each gets what it asked for."""
import threading

import numpy as np
import pytest

import mpm2d
import scenes

pytestmark = pytest.mark.gpu

ROUNDS = 60


def in_threads(jobs):
    """Runs every job ROUNDS times in a thread of its own; the jobs' failures."""
    failed = []

    def loop(k, job):
        for _ in range(ROUNDS):
            try:
                if not job():
                    failed.append(k)
                    return
            except Exception as e:      # reported by the caller
                failed.append((k, repr(e)))
                return
    threads = [threading.Thread(target=loop, args=(k, j)) for k, j in jobs.items()]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return failed


def same(read, want):
    return lambda: np.array_equal(read(), want)


FIELDS = ["x", "y", "vx", "vy", "sxx", "syy"]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_fields(precision):
    sim = mpm2d.Simulation(scenes.box_fill(cells=192, material="isolin"), precision=precision)   # chunks of their own
    sim.step(5)
    want = {k: sim.get(k) for k in FIELDS}
    assert all(not np.array_equal(want[a], want[b]) for a, b in zip(FIELDS, FIELDS[1:]))
    assert in_threads({k: same(lambda k=k: sim.get(k), want[k]) for k in FIELDS}) == []
    frame = {("frame", k): (lambda k=k: np.array_equal(sim.get_frame([k, "y"])[k], want[k])) for k in FIELDS}
    assert in_threads(frame) == []
    sim.close()


def test_gradients():
    sc = scenes.column(Nx=65, Ny=33, h=1.0 / 64, width=0.5, height=0.4, material="isolin", dt=1e-5)
    sim = mpm2d.Simulation(sc)
    sim.adj_forward_tape(4, 2)
    sim.adj_backward(np.linspace(0.0, 1.0, sim.n), np.ones(sim.n))
    names = ["x", "y", "vx", "vy", "v", "sxx"]
    want = {k: sim.adj_state(k) for k in names}
    assert in_threads({k: same(lambda k=k: sim.adj_state(k), want[k]) for k in names}) == []
    sim.close()


def test_sorts():
    sim = mpm2d.Simulation(scenes.box_fill(cells=64, material="isolin"))
    sim.step(5)
    keys, perm, start = sim.get_sort()
    elem, active = sim.get_map()
    assert np.array_equal(perm, np.argsort(np.where(active != 0, elem, sim.ne), kind="stable"))

    def read():
        k, p, s = sim.get_sort()
        return np.array_equal(k, keys) and np.array_equal(p, perm) and np.array_equal(s, start)
    assert in_threads({k: read for k in range(6)}) == []
    sim.close()
