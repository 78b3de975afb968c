"""The multigrid solve's conversions between its FP32 V-cycle and the FP64 outer
iteration (tests/cuda/mg_words_check.cu, built here with nvcc): exact for normal
values, and infinities and NaN carried through."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def words(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = str(tmp_path_factory.mktemp("words") / "libmg_words_check.so")
    src = os.path.join(ROOT, "tests", "cuda", "mg_words_check.cu")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "include"), "-shared",
                    "-Xcompiler", "-fPIC", "-o", out, src], check=True, capture_output=True)
    lib = C.CDLL(out)
    lib.widen.argtypes = [C.c_longlong, C.c_void_p, C.c_int, C.c_void_p]
    lib.narrow.argtypes = [C.c_longlong, C.c_void_p, C.c_int, C.c_void_p]
    return lib


def convert(words, name, x, e):
    import torch
    d = torch.as_tensor(x, device="cuda")
    out = torch.empty(d.numel(), dtype=torch.float64 if name == "widen" else torch.float32, device="cuda")
    assert getattr(words, name)(d.numel(), d.data_ptr(), e, out.data_ptr()) == 0
    return out.cpu().numpy()


@pytest.mark.parametrize("e", [-500, -1, 0, 1, 77, 500])
def test_wide_is_exact_and_carries_non_finite(words, e):
    bits = np.random.default_rng(e + 1000).integers(0, 1 << 32, 1 << 20, dtype=np.uint64).astype(np.uint32)
    edge = np.array([0, 0x80000000, 1, 0x007fffff, 0x00800000, 0x80800000, 0x7f7fffff, 0xff7fffff, 0x3f800000,
                     0x7f800000, 0xff800000, 0x7fc00000, 0xffc00000, 0x7f800001], dtype=np.uint32)
    f = np.concatenate([edge, bits]).view(np.float32)
    with np.errstate(all="ignore"):
        want = np.ldexp(f.astype(np.float64), e)
    want[np.abs(f) < np.float32(2.0 ** -126)] = 0.0        # subnormals and zeros
    got = convert(words, "widen", f, e)
    assert np.array_equal(np.isnan(got), np.isnan(f))
    ok = ~np.isnan(f)
    assert np.array_equal(got[ok], want[ok])


@pytest.mark.parametrize("e", [-500, -1, 0, 1, 77, 500])
def test_narrow_rounds_once_and_carries_non_finite(words, e):
    rng = np.random.default_rng(e + 2000)
    x = np.ldexp(rng.uniform(-2.0, 2.0, 1 << 20), rng.integers(-140, 127, 1 << 20) - e)
    x = np.concatenate([[0.0, -0.0, np.inf, -np.inf, np.nan, np.ldexp(1.0, -126 - e), np.ldexp(1.0, 128 - e), np.ldexp(-1.5, 300 - e),
                         np.ldexp(1.0 + 2.0 ** -24, -e),
                         np.ldexp(1.0 + 3 * 2.0 ** -24, -e)], x])
    s = np.ldexp(x, e)
    with np.errstate(all="ignore"):
        want = s.astype(np.float32)
    want[np.abs(s) < 2.0 ** -126] = 0.0
    got = convert(words, "narrow", x, e)
    assert np.array_equal(np.isnan(got), np.isnan(x))
    ok = ~np.isnan(x)
    assert np.array_equal(got[ok], want[ok])
