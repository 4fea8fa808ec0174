"""Joining float pairs by an FP64 addition (df_join2, the gate kernels) is at
no magnitude less accurate than by integers (df_join): per power of two, the
largest relative error over random pairs.  Compiled for the host from the
kernels' header."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "qcware_unitair_gb300" / "csrc"


@pytest.fixture(scope="module")
def join(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    out = tmp_path_factory.mktemp("dfj") / "libdfj.so"
    subprocess.run([cxx, "-O2", "-ffp-contract=off", "-shared", "-fPIC",
                    f"-I{CSRC}", str(HERE / "native" / "dfloat_join.cpp"),
                    "-o", str(out)], check=True)
    fn = ctypes.CDLL(str(out)).dfj_join

    def call(hi, lo, hi2, lo2):
        n = len(hi)
        re = np.stack([hi, lo], 1).astype(np.float32).copy()
        im = np.stack([hi2, lo2], 1).astype(np.float32).copy()
        a, b = np.empty((n, 2)), np.empty((n, 2))
        fn(re.ctypes.data_as(ctypes.c_void_p),
           im.ctypes.data_as(ctypes.c_void_p), n,
           a.ctypes.data_as(ctypes.c_void_p),
           b.ctypes.data_as(ctypes.c_void_p))
        return a, b

    return call


def pairs(rng, e, n):
    """hi in [2^e, 2^(e + 1)), lo within half an ulp of it, both signs."""
    hi = (2.0 ** e * rng.uniform(1, 2, n)).astype(np.float32)
    lo = (hi.astype(np.float64) * rng.uniform(-1, 1, n) * 2.0 ** -25).astype(
        np.float32)
    sign = rng.choice([-1, 1], n).astype(np.float32)
    return hi * sign, lo


@pytest.mark.parametrize("other", [0, -60])
def test_no_magnitude_is_worse(join, other):
    """``other``: the exponent of the component joined beside it."""
    rng = np.random.default_rng(7)
    for e in range(-126, 61):
        hi, lo = pairs(rng, e, 2000)
        hi2, lo2 = pairs(rng, other, 2000)
        exact = hi.astype(np.float64) + lo.astype(np.float64)
        whole, added = join(hi, lo, hi2, lo2)
        ulp = 2.0 ** -52  # of the result's rounding
        was = np.abs(whole[:, 0] / exact - 1).max()
        now = np.abs(added[:, 0] / exact - 1).max()
        assert now <= max(was, ulp), e
        want = hi2.astype(np.float64) + lo2.astype(np.float64)
        assert np.abs(added[:, 1] / want - 1).max() <= ulp


def test_zero_and_subnormal(join):
    hi = np.array([0.0, -0.0, 2.0 ** -127, -2.0 ** -140, 2.0 ** -126, 1.0],
                  np.float32)
    lo = np.zeros(6, np.float32)
    _, added = join(hi, lo, hi, lo)
    assert np.array_equal(added[:, 0], [0, 0, 0, 0, 2.0 ** -126, 1.0])
    assert np.array_equal(added[:, 0], added[:, 1])
    assert list(np.signbit(added[:, 0])) == [False, True, False, True, False,
                                             False]
