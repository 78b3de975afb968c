"""The multigrid solve's conversions between its FP32 V-cycle and the FP64 outer
iteration (tests/cuda/mg_words_check.cu, built here with nvcc): exact for normal
values, and infinities and NaN carried through.  And its waits for other blocks'
words: a wait that runs out (words that nothing writes, a poll limit of 1024)
returns, sets the spin status, and no total of it passes for a converged one."""
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
                    "-DMPMG_MG_POLL_LIMIT=1024", "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "include"), "-shared",
                    "-Xcompiler", "-fPIC", "-o", out, src], check=True, capture_output=True)
    lib = C.CDLL(out)
    lib.widen.argtypes = [C.c_longlong, C.c_void_p, C.c_int, C.c_void_p]
    lib.narrow.argtypes = [C.c_longlong, C.c_void_p, C.c_int, C.c_void_p]
    lib.wait_block.argtypes = [C.c_void_p, C.c_int, C.c_void_p, C.c_int, C.c_void_p, C.c_uint, C.c_void_p, C.c_void_p]
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


SPIN = 4       # MPMG_DEV_ERR_SPIN


def wait_block(words, nblocks, present, staged=0, staged_present=True, tag=77):
    """One block's gather among nblocks; `present` of the others have published (value c of
    block b: 100 c + b), the rest, and this one's own before it publishes, hold an older tag."""
    import torch
    w = np.zeros((4, nblocks, 2), dtype=np.uint64)
    val = (100.0 * np.arange(4)[:, None] + np.arange(nblocks)[None, :]).view(np.uint64)
    b = np.arange(nblocks)
    tags = np.where((b > 0) & (b <= present), tag, tag - 1).astype(np.uint64)[None, :] << np.uint64(32)
    w[:, :, 0] = tags | (val & np.uint64(0xffffffff))
    w[:, :, 1] = tags | (val >> np.uint64(32))
    s = np.arange(max(staged, 1)).astype(np.float32).view(np.uint32).astype(np.uint64)
    s |= np.uint64((tag if staged_present else tag - 1) << 32)
    dw, ds = (torch.as_tensor(a.view(np.int64).ravel(), device="cuda") for a in (w, s))
    floats = torch.zeros(max(staged, 1), dtype=torch.float32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.zeros(5, dtype=torch.float64, device="cuda")
    assert words.wait_block(dw.data_ptr(), nblocks, ds.data_ptr(), staged, floats.data_ptr(), tag, status.data_ptr(),
                            out.data_ptr()) == 0
    out = out.cpu().numpy()
    return out[:4], bool(out[4]), int(status.item()), floats.cpu().numpy()


@pytest.mark.parametrize("nblocks", [1, 2, 33, 152, 160])
def test_gather_sums_every_block(words, nblocks):
    total, ok, status, floats = wait_block(words, nblocks, nblocks - 1, staged=50)
    others = np.arange(1, nblocks)
    want = [1.0 + c + np.sum(100.0 * c + others) for c in range(4)]     # whole numbers: any order
    assert ok and status == 0 and np.array_equal(total, want)
    assert np.array_equal(floats, np.arange(50))


@pytest.mark.parametrize("nblocks,present", [(2, 0), (33, 31), (160, 0)])
def test_gather_that_runs_out_is_no_result(words, nblocks, present):
    total, ok, status, _ = wait_block(words, nblocks, present)
    assert not ok and status == SPIN
    assert np.isnan(total).all()


@pytest.mark.parametrize("nblocks", [1, 152])
def test_stage_that_runs_out_never_converges(words, nblocks):
    """The words read NaN, and the residual this block publishes is NaN, though every
    block's word arrives."""
    total, ok, status, floats = wait_block(words, nblocks, nblocks - 1, staged=50, staged_present=False)
    assert ok and status == SPIN
    assert np.isnan(floats).all() and np.isnan(total[3])
