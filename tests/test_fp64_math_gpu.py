"""The device paths of the FP64 elementary functions and comparisons (wf_math.cuh) against the host
paths, bit for bit: the FP64 form reproduces the reference's arithmetic only if they agree. The
values cover magnitudes, signs, zeros, subnormals, infinities and NaN, and the quotients nearest to a
rounding boundary (both operands a few ulps from powers of two)."""

import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = ("div", "div_by", "exp", "log", "pow", "jmin", "jmax", "jclamp", "cld", "cbrt", "comparisons")


@pytest.fixture(scope="module")
def probe(gpu_lib, tmp_path_factory):
    from wflow_gb300 import build
    so = tmp_path_factory.mktemp("math") / "libprobe.so"
    src = Path(__file__).with_name("fp64_math_probe.cu")
    subprocess.run([build._nvcc(), *build.ARCH, "-O3", "-std=c++17", "--fmad=false", "-shared", "-Xcompiler",
                    "-fPIC,-ffp-contract=off", "-I", str(build.CSRC), "-o", str(so), str(src)], check=True)
    return C.CDLL(str(so))


def values(kind, n, rng):
    if kind == "wide":
        a, b = (rng.choice([-1.0, 1.0], n) * 10.0 ** rng.uniform(-300, 300, n) for _ in range(2))
    elif kind == "ordinary":
        a, b = (rng.choice([-1.0, 1.0], n) * 10.0 ** rng.uniform(-12, 6, n) for _ in range(2))
    elif kind == "unit":
        a, b = rng.uniform(0.0, 1.0, n), rng.uniform(0.0, 2.0, n)
    elif kind == "near_powers":
        a, b = (np.ldexp(1.0 + rng.integers(-40, 41, n) * 2.0 ** -53, rng.integers(-3, 4, n)) for _ in range(2))
    elif kind == "steps":  # whole and ragged multiples of the unsaturated flow's step
        b = np.full(n, 2e-4)
        a = np.where(rng.random(n) < 0.5, rng.integers(0, 400, n) * 2e-4, rng.uniform(0.0, 0.08, n))
    else:  # special values in all pairs
        s = np.array([0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.2e-308, 1.7e308, -1.7e308, 3600.0,
                      709.0, 710.0, -745.0, -746.0, -708.0, 700.5, -700.5])
        a, b = (x.reshape(-1) for x in np.meshgrid(s, s))
    return np.ascontiguousarray(a, np.float64), np.ascontiguousarray(b, np.float64)


@pytest.mark.parametrize("kind", ["wide", "ordinary", "unit", "near_powers", "steps", "special"])
def test_device_paths_equal_host_paths(probe, kind):
    a, b = values(kind, 200_000, np.random.default_rng(12))
    n = a.size
    host, dev = np.empty((len(NAMES), n)), np.empty((len(NAMES), n))
    p = lambda x: x.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    assert probe.probe_host(p(a), p(b), p(host), C.c_int64(n)) == len(NAMES)
    assert probe.probe_device(p(a), p(b), p(dev), C.c_int64(n)) == 0
    for name, h, d in zip(NAMES, host, dev):
        same = (h == d) | (np.isnan(h) & np.isnan(d))
        assert same.all(), (name, a[~same][:3], b[~same][:3], h[~same][:3], d[~same][:3])
