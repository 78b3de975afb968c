"""mat::exp_small (the volume update's exponential) against 60 decimal digits, over all its
branches: zeros, subnormals, arguments that round away, fixed point below 2^-14, the
polynomial below 2^-9, exp() beyond, and values that are not finite.  Either polynomial is
within a hundredth of a unit in the last place before its last rounding, exp() within one."""
import ctypes as C
import decimal
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def exp_of(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = str(tmp_path_factory.mktemp("exp") / "libexp_check.so")
    src = os.path.join(ROOT, "tests", "cuda", "exp_check.cu")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I", os.path.join(ROOT, "include"), "-shared", "-Xcompiler", "-fPIC", "-o", out, src], check=True,
                   capture_output=True)
    lib = C.CDLL(out)
    dp = C.POINTER(C.c_double)
    lib.exp_of.argtypes = [C.c_int, dp, dp]

    def run(x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        y = np.empty_like(x)
        assert lib.exp_of(x.size, x.ctypes.data_as(dp), y.ctypes.data_as(dp)) == 0
        return y
    return run


def errors(x, y):
    """|y - e^x| in units of e^x's last place."""
    with decimal.localcontext() as c:
        c.prec = 60
        out = []
        for a, b in zip(x.tolist(), y.tolist()):
            want = decimal.Decimal(a).exp()
            ulp = decimal.Decimal(2) ** (-53 if want < 1 else -52)
            if want >= 2 or want < decimal.Decimal("0.5"):
                ulp = decimal.Decimal(float(np.spacing(float(want))))
            out.append(float(abs(decimal.Decimal(b) - want) / ulp))
    return np.array(out)


def around(e):
    """The doubles next to 2^e, with signs."""
    a = 2.0 ** e
    near = [a]
    for d in (np.inf, 0.0):
        b = a
        for _ in range(3):
            b = np.nextafter(b, d)
            near.append(b)
    return np.array(near + [-v for v in near])


def test_edges(exp_of):
    x = np.concatenate([[0.0, -0.0, 5e-324, -5e-324, 2.0 ** -1022, -2.0 ** -1022]] +
                       [around(e) for e in (-1000, -64, -63, -62, -61, -55, -54, -53, -52, -40, -15, -14, -13, -10)])
    assert errors(x, exp_of(x)).max() <= 0.51
    x = np.concatenate([around(-9), around(-8), [1.0, -1.0, 3.0, -3.0]])
    assert errors(x, exp_of(x)).max() <= 1.0
    y = exp_of([np.inf, -np.inf, np.nan, 1e4, -1e4])
    assert y[0] == np.inf and y[1] == 0.0 and np.isnan(y[2]) and y[3] == np.inf and y[4] == 0.0


@pytest.mark.parametrize("low, high", [(-70, -50), (-50, -30), (-30, -14), (-16, -9)])
def test_ranges(exp_of, low, high):
    rng = np.random.default_rng(-high)
    x = np.exp2(rng.uniform(low, high, 20000)) * rng.choice([-1, 1], 20000)
    assert errors(x, exp_of(x)).max() <= 0.51
