"""Calls that allocate on first need, with an allocator that fails (a build of
the library whose mpmg_api.cu takes tests/cuda/fake_alloc.h's): they report it or
do without, and the next call works."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def variant(tmp_path_factory):
    import mpm2d
    import mpmg_build
    mpm2d.lib()                # the library's objects, up to date
    tmp = tmp_path_factory.mktemp("fake")
    obj, out = str(tmp / "api.o"), str(tmp / "libmpm_gb300_fake.so")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc] + mpmg_build.ARCH + mpmg_build.NVCC_FLAGS +
                   ["-include", os.path.join(ROOT, "tests", "cuda", "fake_alloc.h"), "-c",
                    os.path.join(PKG, "csrc", "mpmg_api.cu"), "-o", obj], check=True, capture_output=True)
    objs = [os.path.join(mpmg_build.OUT, os.path.splitext(s)[0] + ".o") for s in mpmg_build.CU_SOURCES
            if s != "mpmg_api.cu"]
    subprocess.run([nvcc] + mpmg_build.ARCH + ["-shared", "-o", out, obj] + objs + ["-lcudart", "-ldl", "-lpthread"],
                   check=True, capture_output=True)
    return out


@pytest.fixture
def fake(variant, monkeypatch):
    """mpm2d on the variant; its simulations have to be closed before the test ends."""
    import mpm2d
    monkeypatch.setattr(mpm2d, "_lib", None)
    monkeypatch.setattr(mpm2d._build, "build", lambda *a, **k: variant)
    lib = mpm2d.lib()
    device, pinned = (C.c_int.in_dll(lib, "mpmg_test_fail_" + k) for k in ("device", "pinned"))
    device.value, pinned.value = -1, 0
    yield mpm2d, device, pinned
    device.value, pinned.value = -1, 0


def test_sort_without_memory_then_with(fake):
    import scenes
    mpm2d, device, _ = fake
    sim = mpm2d.Simulation(scenes.config1())
    sim.step(3)
    for fail_at in range(6):                    # the sort's six arrays
        device.value = fail_at
        with pytest.raises(mpm2d.MpmError, match="out of device memory"):
            sim.get_sort()
    device.value = -1
    sim.step(1)                                 # no error left behind
    elem, active = sim.get_map()
    want = np.argsort(np.where(active != 0, elem, sim.ne), kind="stable")
    keys, perm, start = sim.get_sort()
    assert np.array_equal(perm, want)
    assert np.array_equal(start, np.searchsorted(keys, np.arange(sim.ne + 1)))
    sim.close()


def test_read_back_without_pinned_memory(fake):
    import scenes
    mpm2d, _, pinned = fake
    sim = mpm2d.Simulation(scenes.config1())
    sim.step(3)
    pinned.value = 1
    first = sim.get_frame(["x", "vy", "sxx"])
    again = sim.get("vy")
    pinned.value = 0
    later = sim.get_frame(["x", "vy", "sxx"])   # through the pinned chunks
    for k in first:
        assert np.array_equal(first[k], later[k]), k
    assert np.array_equal(again, first["vy"])
    sim.close()
