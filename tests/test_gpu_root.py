"""The FP64 step's square root, quotients and product against the IEEE operations, bit
for bit (tests/cuda/root_check.cu, built here with nvcc): mat::root and
mat::quot (one FP64 operation and a rounding in units of the last place, with
the folded powers of two), mat::dvd_const and mat::imul (integer
arithmetic), on random operands, next to midpoints of two doubles,
next to powers of two, on short significands and on arbitrary bit patterns."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

N = 1 << 24


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = str(tmp_path_factory.mktemp("root") / "libroot_check.so")
    src = os.path.join(ROOT, "tests", "cuda", "root_check.cu")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "include"), "-shared",
                    "-Xcompiler", "-fPIC", "-o", out, src], check=True, capture_output=True)
    fn = C.CDLL(out).check_op
    fn.argtypes = [C.c_int, C.c_int, C.c_int, C.c_double, C.c_longlong, C.c_ulonglong,
                   C.POINTER(C.c_ulonglong), C.POINTER(C.c_double)]

    def run(op, kind, span, b=1.0, n=N, seed=1):
        bad, ex = C.c_ulonglong(), (C.c_double * 4)()
        assert fn(op, kind, span, b, n, seed, C.byref(bad), ex) == 0
        assert bad.value == 0, (op, kind, span, b, bad.value, [v.hex() for v in ex])
    return run


@pytest.mark.parametrize("kind,span", [(0, 60), (0, 1000), (1, 1), (2, 60), (3, 60), (16, 60), (18, 60), (19, 60),
                                       (20, 60), (24, 60), (28, 60)])
def test_root_quotient_product_equal_ieee(check, kind, span):
    check(0, kind, min(span, 400) if kind & 16 else span)
    for kb in (0, 4, 8, 12) if kind < 4 else (0,):
        check(1, kind | kb, min(span, 400) if kind & 16 else span)
        if kind < 4:
            check(3, kind | kb, span)   # kinds 2 and 3 have ties


@pytest.mark.parametrize("kind", [0, 2, 3, 16])
def test_constant_divisors_equal_ieee(check, kind):
    rng = np.random.default_rng(7)
    fixed = [3.0, 1e6 / 2.6, 2e-6, 5e-6, 1e-5, 2450.0, 5.3e-4, 0.005, 1.0, 0.5, 2.0 - 2.0**-52, 1.0 + 2.0**-52,
             float.fromhex("0x1.898b63fe31d03p+0"), float.fromhex("0x1.da43ea185cc8fp-20"),
             2.0**-401, 2.0**401, 1e-310, 0.0, float("inf"), float("nan")]   # the last six: the compiler's division
    for i, b in enumerate(fixed + list(np.exp(rng.uniform(-20, 20, 40)) * rng.choice([-1, 1], 40))):
        check(2, kind, 60, float(b), n=1 << 21, seed=i)
    check(2, 1, 1, 3.0)   # any bit pattern
