"""rsqrt64.cuh by itself: the seed, x^(-1/2) and x^(-3/2) against 64-bit mantissas on the host, over random exponents and both
ends of the range, and which inputs are in it.

Bounds (relative). Seed: |1 - x y^2| < 2^-18, y of at most 21 significant bits. Truncation of the series: 5/16 and 35/16 times
|e|^3 < 2^-54, below 2^-52 together with the next terms; the last rounding 2^-53, x^(-3/2) one more for y^3; the others act
on terms of 2^-18 and less and stay below 2^-60 in all."""

import ctypes
import shutil
import subprocess

import numpy as np
import pytest

from grasph2_b200 import build
from test_dependent_launches import CSRC

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    import os
    nvcc = build.nvcc()
    assert shutil.which(nvcc) or os.path.exists(nvcc)
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp", "rsqrt64_check.cu")
    lib = str(tmp_path_factory.mktemp("rsqrt64") / "librsqrt64_check.so")
    subprocess.run([nvcc] + build.ARCH + ["-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I", CSRC, src, "-o", lib],
                   check=True)
    f = ctypes.CDLL(lib).rsqrt64_check

    def call(x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        out, flags = np.empty((3, len(x))), np.empty(len(x), dtype=np.int32)
        p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
        assert f(p(x), p(out), p(flags), len(x)) == 0
        return out, flags
    return call


def test_errors(run):
    rng = np.random.default_rng(1)
    n = 1 << 20
    x = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-600, 600, n))
    x[:4] = [2.0 ** -600, np.nextafter(2.0 ** 600, 0), 1.0, np.nextafter(1.0, 2)]
    (seed, half, cube), ok = run(x)
    assert ok.all()
    xl = x.astype(np.longdouble)
    r = np.sqrt(xl)
    y = seed.astype(np.longdouble)
    assert np.abs(1 - xl * y * y).max() < 2.0 ** -18
    assert not (seed.view(np.uint64) & np.uint64((1 << 32) - 1)).any()  # 20 bits behind the leading one
    assert np.abs(half * r - 1).max() <= 2.0 ** -52 + 2.0 ** -53 + 2.0 ** -60
    assert np.abs(cube * (xl * r) - 1).max() <= 2.0 ** -52 + 2.0 ** -52 + 2.0 ** -60


def test_range(run):
    inside = [2.0 ** -600, np.nextafter(2.0 ** 600, 0), 1.0]
    outside = [2.0 ** 600, np.nextafter(2.0 ** -600, 0), 0.0, -0.0, 5e-324, -1.0, -2.0 ** -600, np.inf, -np.inf, np.nan]
    _, ok = run(np.array(inside + outside))
    assert ok[:3].all() and not ok[3:].any()
