"""The split form's kinematic-wave solve (wf_kw_ff.cuh) against 64-bit roots over the discharges, cell
lengths, steps and roughnesses of a catchment, from previous discharges far below and far above the new one,
next to it and none. The bar on Q, 1e-12, is the solve's error bound of 7e-13 (stated there) and the
roundings of the double-FP32 products."""

import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def probe(gpu_lib, tmp_path_factory):
    from wflow_gb300 import build
    so = tmp_path_factory.mktemp("solve") / "libsolve.so"
    src = Path(__file__).with_name("split_solve_probe.cu")
    subprocess.run([build._nvcc(), *build.ARCH, "-O3", "-std=c++17", "-prec-div=false", "-shared", "-Xcompiler",
                    "-fPIC,-ffp-contract=off", "-I", str(build.CSRC), "-I", str(build.REPO_ROOT / "include"),
                    "-o", str(so), str(src)], check=True)
    return C.CDLL(str(so))


def pair(x):
    """x as a double-FP32 pair holds it"""
    h = x.astype(np.float32).astype(np.float64)
    return h + (x - h).astype(np.float32).astype(np.float64)


def root(cterm, a, b):
    u = np.minimum(np.cbrt(cterm / b), (cterm / a) ** 0.2)
    for _ in range(60):
        u = u - (u ** 3 * (a * u * u + b) - cterm) / (u * u * (5.0 * a * u * u + 3.0 * b))
    return u


@pytest.mark.parametrize("start", ["far", "near", "none"])
def test_discharge(probe, start):
    rng, n = np.random.default_rng(16), 1_000_000
    dt_dx = pair(10.0 ** rng.uniform(-1.0, 3.0, n))
    alpha = (10.0 ** rng.uniform(-1.5, 1.5, n)).astype(np.float32).astype(np.float64)
    u = 10.0 ** rng.uniform(-2.4, 1.0, n)  # Q from 1e-12 to 1e5 m3/s
    cterm = pair(u ** 3 * (dt_dx * u * u + alpha))
    u = root(cterm, dt_dx, alpha)
    if start == "far":
        u_prev = np.maximum(u * 10.0 ** rng.uniform(-3.0, 3.0, n), 1e-6)
    elif start == "near":
        u_prev = u * (1.0 + rng.choice([-1.0, 1.0], n) * 10.0 ** rng.uniform(-8.0, -1.0, n))
    else:
        u_prev = np.zeros(n)
    x = np.ascontiguousarray(np.stack([cterm, dt_dx, alpha, u_prev]))
    out = np.empty((2, n))
    p = lambda v: v.ctypes.data_as(C.c_void_p)  # noqa: E731
    assert probe.solve_device(p(x), p(out), C.c_int64(n)) == 0
    err = np.abs(out[1] - u ** 5) / u ** 5
    print(f"{start}: largest error of Q {err.max():.2e}, mean square {np.sqrt((err ** 2).mean()):.2e}")
    assert err.max() <= 1e-12, (err.max(), x[:, err.argmax()])
