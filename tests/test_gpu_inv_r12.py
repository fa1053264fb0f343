"""1/r12 from r12^2 in FP64 (invR12 of csrc/common.cuh), which every FP64 kernel value hangs on, against 80-bit 1/sqrt(x).

The step's own rounding is at most 3/2 2^-53 of the result: 2^-53 of e = 1 - x y^2 enters halved, the last addition rounds once
more; the series' next term is below that of the last place.  The bar is 2^-52, over every exponent of a normal
number and over the r12^2 of the grids.  Zero and what the hardware estimate takes for zero (subnormal
numbers) give 0, the rule for coincident points."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from tcscf_b200 import build

pytestmark = pytest.mark.gpu

SRC = Path(__file__).resolve().parent / "cpp" / "inv_r12.cu"


@pytest.fixture(scope="module")
def inv_r12(tmp_path_factory):
    if not Path(build.NVCC).exists():
        pytest.skip("needs nvcc")
    so = tmp_path_factory.mktemp("inv_r12") / "inv_r12.so"
    res = subprocess.run([build.NVCC, *build.ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I", str(build.CSRC), str(SRC), "-o", str(so)],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-4000:]
    f = C.CDLL(str(so)).inv_r12
    p = np.ctypeslib.ndpointer(np.float64, flags="C_CONTIGUOUS")
    f.argtypes, f.restype = [C.c_int64, p, p], C.c_int

    def call(x):
        y = np.full_like(x, np.nan)
        assert f(x.size, x, y) == 0
        return y

    return call


def _relative_error(x, y):
    assert np.finfo(np.longdouble).nmant >= 63
    return float(np.abs(y.astype(np.longdouble) * np.sqrt(x.astype(np.longdouble)) - 1).max())


def test_every_exponent(inv_r12):
    rng = np.random.default_rng(1)
    exps = np.arange(-1022, 1024)
    m = np.concatenate([[1.0, np.nextafter(1, 2), np.nextafter(2, 1), 1.5], rng.uniform(1, 2, 1020)])
    x = np.ldexp(m[None, :], exps[:, None]).ravel()
    err = _relative_error(x, inv_r12(x))
    print(f"largest relative error {err * 2**53:.3f} x 2^-53")
    assert err <= 2.0 ** -52


def test_the_range_of_the_grids(inv_r12):
    x = 10.0 ** np.random.default_rng(2).uniform(-24, 12, 1 << 22)
    assert _relative_error(x, inv_r12(x)) <= 2.0 ** -52


def test_coincident_points(inv_r12):
    tiny = np.finfo(np.float64).tiny
    x = np.array([0.0, 5e-324, 2.0 ** -1060, 2.0 ** -1043, 2.0 ** -1042, 2.0 ** -1041, 2.0 ** -1030, np.nextafter(tiny, 0), tiny])
    y = inv_r12(x)
    assert (y[:-1] == 0).all(), y
    assert y[-1] == 2.0 ** 511
