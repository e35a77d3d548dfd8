"""The force terms' square roots over the whole normal range (tests/cuda/roots.cu, built
with the package's flags) against 80-bit values and the CUDA library's."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "ladds_b200", "csrc")


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    from ladds_b200 import build

    out = str(tmp_path_factory.mktemp("roots") / "libroots.so")
    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    r = subprocess.run([nvcc, *build.NVCC_ARCH, *build.NVCC_FLAGS, "-shared", "-I", CSRC, "-o", out,
                        os.path.join(HERE, "cuda", "roots.cu")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return out


def test_roots_build(library):
    assert os.path.exists(library)


def ulps(got, want):
    """Distance of binary64 values from 80-bit ones in units of the last place."""
    near = want.astype(np.float64)
    return np.abs(got.astype(np.longdouble) - want) / np.spacing(near).astype(np.longdouble)


@pytest.mark.gpu
def test_roots_over_the_normal_range(library):
    """rsqrtOf: the series leaves out 2^-77 and its products round at 2^-72 of the result, so
    the last rounding is all of its error: half a unit, and 2^-11 units for the 80-bit
    value's own rounding; bound 0.501.  sqrtOf = x rsqrtOf(x): half a unit for its own rounding
    and the reciprocal's half unit, up to one here; bound 1.5.  The library's functions
    are named to be within 1 and 0.5 units, so the roots differ by less than 1.6."""
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(1)
    lo, hi = np.finfo(np.float64).tiny, np.finfo(np.float64).max
    near = (np.arange(-200_000, 200_001) * 2.0**-52)
    x = np.concatenate([
        rng.uniform(1.0, 4.0, 2_000_000),  # both exponent parities
        np.ldexp(rng.uniform(1.0, 2.0, 2_000_000), rng.integers(-1022, 1024, 2_000_000)),
        1.0 + np.abs(near), 2.0 - np.abs(near) / 2, 2.0 + 2 * np.abs(near), 4.0 - 2 * np.abs(near), 4.0 + 4 * np.abs(near),
        np.geomspace(1e2, 1e18, 500_000),  # squared distances
        [lo, np.nextafter(lo, 1.0), hi, np.nextafter(hi, 0.0)]])
    roots = ctypes.CDLL(library).roots
    roots.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
    out = np.zeros((4, len(x)))
    assert roots(x.ctypes.data, len(x), out.ctypes.data) == 0
    root = np.sqrt(x.astype(np.longdouble))
    assert np.finfo(np.longdouble).nmant >= 63
    assert np.max(ulps(out[0], 1 / root)) < 0.501
    assert np.max(ulps(out[1], root)) < 1.5
    assert np.max(np.abs(out[0] - out[2]) / np.spacing(out[2])) <= 1.0
    assert np.max(np.abs(out[1] - out[3]) / np.spacing(out[3])) <= 1.0
    # outside it: what the force terms' comments say
    odd = np.array([0.0, np.inf, np.nan, lo / 4, -1.0])
    out = np.zeros((4, len(odd)))
    assert roots(odd.ctypes.data, len(odd), out.ctypes.data) == 0
    assert np.all(np.isnan(out[0, :3]))
    assert out[1, 0] == 0.0 and np.isnan(out[1, 2]) and out[1, 3] == lo / 4 and out[1, 4] == -1.0
