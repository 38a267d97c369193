"""The FP64 reciprocal square root and exponential of the panel-pair kernels (csrc/fastmath.cuh) against extended precision
and CUDA's own functions, over the ranges that they are written for.

u = 2^-53.  rsqrt_pos: x y^2 is formed with one rounding (u/2 in the result), the result with another (u), and the
truncation is 5/16 (2^-19)^3 = 0.02 u from a seed good to 2^-20: 1.6 u.  exp_tab: the table's values and the last
operation are rounded (2 u), the Taylor polynomial is truncated by 0.0054^6 / 720 = 0.32 u: 2.4 u.  CUDA's functions are
within 1 ulp = 2 u.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu
U = 2.0 ** -53
LD = np.longdouble


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fastmath") / "probe.so")
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                    "-I", os.path.join(ROOT, "cuda-fabipb_b200", "csrc"), os.path.join(ROOT, "tests", "fastmath_probe.cu"),
                    "-o", so], check=True)
    f = C.CDLL(so).fastmath_probe

    def run(x, s):
        x, s = (np.ascontiguousarray(v, dtype=np.float64) for v in (x, s))
        out = np.empty((4, len(x)))
        ptr = [v.ctypes.data_as(C.c_void_p) for v in (x, s, out)]
        assert len(x) == len(s) and f(len(x), *ptr) == 1
        return out
    return run


def rel(a, exact):
    return np.abs((a.astype(LD) - exact) / exact).max()


def test_rsqrt_pos(probe):
    rng = np.random.default_rng(1)
    power = 4.0 ** np.arange(-500, 500)
    x = np.concatenate([np.exp(rng.uniform(np.log(1e-300), np.log(1e300), 1 << 20)), rng.uniform(1, 4, 1 << 20),
                        power, np.nextafter(power, 0), np.nextafter(power, np.inf), 2 * power])
    own, lib = probe(x, np.zeros(len(x)))[:2]
    exact = 1 / np.sqrt(x.astype(LD))
    assert rel(own, exact) <= 1.6 * U
    assert np.abs(own / lib - 1).max() <= 4 * U   # 1.6 u and 2 u, and the quotient's own rounding


def test_exp_tab(probe):
    rng = np.random.default_rng(2)
    half = -(np.arange(0, 65344, 7) + 0.5)   # ends of the table's intervals
    s = np.concatenate([-np.exp(rng.uniform(np.log(1e-12), np.log(65343), 1 << 20)), rng.uniform(-200, 0, 1 << 20), half,
                        np.nextafter(half, 0), np.nextafter(half, -1e9), -np.arange(0.0, 65345.0), [0.0, -0.0, -5e-324]])
    own, lib = probe(np.ones(len(s)), s)[2:]
    exact = np.exp2(s.astype(LD) / 64)
    assert rel(own, exact) <= 2.4 * U
    assert np.abs(own / lib - 1).max() <= 5 * U


def test_exp_tab_ends(probe):
    """Exactly 1 at 0; 2^-1021 from -64 * 1021 down; a NaN stays one."""
    s = np.array([0.0, -0.0, -65344.0, -65345.0, -65408.0, -1e6, -1e300, -np.inf, np.nan])
    own = probe(np.ones(len(s)), s)[2]
    assert (own[:2] == 1).all() and (own[2:8] == 2.0 ** -1021).all() and np.isnan(own[8])
