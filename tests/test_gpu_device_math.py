"""rcp3 (ocfd_device.cuh) and exp2_tab (ocfd_exp2.cuh) against 64-bit division and an extended-precision
exponential, over their exponents and at the edges of their ranges.

Bounds: rcp3's series leaves e^3 <= 2^-60 of the approximation's error e <= 2^-20, so its last rounding
decides: at most one unit in the last place from the correctly rounded quotient. exp2_tab adds the table's
rounding (2^-53), the polynomial's remainder (4e-17) and the last rounding (2^-53): 2.6e-16, and a few
hundredths of that for the roundings of the small term.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["false", "true"], ids=["exact", "contracted"])
def device_math(request, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("math") / "device_math.so")
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-gencode", "arch=compute_100a,code=sm_100a",
                    "-O3", "--fmad=" + request.param, "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-I", os.path.join(ROOT, "opencfd-comb_b200", "csrc"), "-o", so, os.path.join(HERE, "device_math.cu")],
                   check=True, timeout=300)
    fn = C.CDLL(so).device_math
    P = C.POINTER(C.c_double)

    def run(x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        out = np.empty((2, x.size))
        assert fn(x.size, x.ctypes.data_as(P), out[0].ctypes.data_as(P), out[1].ctypes.data_as(P)) == 0
        return out
    return run


def test_reciprocal(device_math):
    rng = np.random.default_rng(0)
    m = np.concatenate([[1.0, 1.0 + 2.0 ** -52, 1.5, 2.0 - 2.0 ** -52], rng.uniform(1.0, 2.0, 300)])
    x = np.ldexp(m[:, None], np.arange(-1022, 1022)[None, :]).ravel()
    x = np.concatenate([x, -x])
    got, want = device_math(x)[0], 1.0 / x
    assert (np.abs(got - want) <= np.spacing(np.abs(want))).all()
    assert np.isnan(device_math([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324])[0]).all()
    assert (device_math(np.ldexp([1.0, 1.9], 1023))[0] == 0.0).all()


def test_exponential(device_math):
    rng = np.random.default_rng(1)
    j = np.arange(-64 * 1021, 64 * 1021, 97) / 64.0
    half = 1.0 / 128.0
    x = np.concatenate([j, j + half, j - half, np.nextafter(j + half, 0.0), rng.uniform(-1021.0, 1022.0, 100000),
                        rng.uniform(-1e-3, 1e-3, 1000), [0.0, 1022.0, -1022.0]])
    got, want = device_math(x)[1], np.exp2(x.astype(np.longdouble))
    assert (np.abs(got - want) <= 2.8e-16 * want).all()
    big = device_math([1100.0, 1e6, -1100.0, -1e6])[1]  # beyond the normal range: held at its ends
    assert (big[:2] >= 2.0 ** 1022).all() and np.isfinite(big[:2]).all()
    assert (big[2:] > 0.0).all() and (big[2:] <= 2.0 ** -1021).all()
    assert np.isnan(device_math([np.nan])[1]).all()
