"""Device paths against host paths to the last bit, signs of zeros included: the elementary functions and
comparisons of wf_math.cuh, quotients with the reciprocals that the kernels use, the edge flows of the
local-inertial schemes, and what a chain end publishes."""

import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from test_fp64_math_gpu import NAMES, probe, values  # noqa: F401 (probe: a fixture)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bits(gpu_lib, tmp_path_factory):
    from wflow_gb300 import build
    so = tmp_path_factory.mktemp("bits") / "libbits.so"
    src = Path(__file__).with_name("fp64_bits_probe.cu")
    subprocess.run([build._nvcc(), *build.ARCH, "-O3", "-std=c++17", "--fmad=false", "-shared", "-Xcompiler",
                    "-fPIC,-ffp-contract=off", "-I", str(build.CSRC), "-I", str(build.REPO_ROOT / "include"),
                    "-o", str(so), str(src)], check=True)
    return C.CDLL(str(so))


def differ(h, d):
    return (h.view(np.uint64) != d.view(np.uint64)) & ~(np.isnan(h) & np.isnan(d))


def call(f, x, rows, n):
    out = np.empty((rows, n), np.float64 if x.dtype == np.float64 else x.dtype)
    assert f(x.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p), C.c_int64(n)) == 0
    return out


@pytest.mark.parametrize("kind", ["wide", "ordinary", "unit", "near_powers", "steps", "special"])
def test_functions(probe, kind):  # noqa: F811
    a, b = values(kind, 200_000, np.random.default_rng(13))
    n = a.size
    host, dev = np.empty((len(NAMES), n)), np.empty((len(NAMES), n))
    p = lambda x: x.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    assert probe.probe_host(p(a), p(b), p(host), C.c_int64(n)) == len(NAMES)
    assert probe.probe_device(p(a), p(b), p(dev), C.c_int64(n)) == 0
    for name, h, d in zip(NAMES, host, dev):
        bad = differ(h, d)
        assert not bad.any(), (name, a[bad][:3], b[bad][:3], h[bad][:3], d[bad][:3])


def hard_quotients(n, rng):
    """Quotients next to the middle of two values: with integers m_b and q of 53 bits, a such that
    2^k a = (2 q + 1) m_b +- 1, for divisors whose mantissa spans [1, 2) and its upper end."""
    a, b = [], []
    for i in range(n):
        top = 2 ** 53 - int(2.0 ** rng.uniform(0, 50)) if i % 2 else int(rng.integers(2 ** 52, 2 ** 53))
        mb = max(top | 1, 2 ** 52 + 1)
        # (2 q + 1) m_b = 1 or -1 (mod 2^53): 2 q + 1 is the inverse, which is odd
        odd = pow(mb, -1, 2 ** 54)
        for s in (odd, 2 ** 54 - odd):
            num = s * mb + (-1 if (s * mb) % 2 ** 54 == 1 else 1)
            ma = num >> 54
            if num % 2 ** 54 == 0 and 2 ** 52 <= ma < 2 ** 53:
                a.append(float(ma))
                b.append(float(mb))
    return np.array(a), np.array(b)


def test_quotients(bits):
    rng = np.random.default_rng(14)
    parts = [values(k, 100_000, rng) for k in ("wide", "ordinary", "unit", "near_powers", "special")]
    parts.append(hard_quotients(300_000, rng))
    assert parts[-1][0].size > 100_000
    ab = np.ascontiguousarray(np.stack([np.concatenate(x) for x in zip(*parts)]))
    n = ab.shape[1]
    host, dev = call(bits.quotients_host, ab, 3, n), call(bits.quotients_device, ab, 3, n)
    for k in range(3):
        bad = differ(host[k], dev[k])
        assert not bad.any(), (k, bad.sum(), ab[:, bad][:, :3], host[k][bad][:3], dev[k][bad][:3])


@pytest.mark.parametrize("decades", [(-3.0, 1.0), (-12.0, -3.0), (-32.0, -20.0)])
def test_edge_flows(bits, decades):
    # depths from the usual ones down to those whose limit of the flow leaves FP32's range; without
    # friction and slope the discharge stays what it was, from the critical one to a part in 10^6 of it
    rng, n = np.random.default_rng(15), 400_000
    hf, w = 10.0 ** rng.uniform(*decades, n), 10.0 ** rng.uniform(-1, 2, n)
    limit = w * hf * np.sqrt(9.80665 * hf)
    q0 = rng.choice([-1.0, 1.0], n) * limit * (1.0 + rng.choice([-1.0, 1.0], n) * 10.0 ** rng.uniform(-6, 0, n))
    still = rng.random(n) < 0.5
    zs0 = np.where(still, 0.0, rng.uniform(0, 10, n))
    zs1 = np.where(still, 0.0, zs0 + rng.uniform(-1, 1, n) * hf)
    x = np.ascontiguousarray(np.stack([q0, zs0, zs1, hf, w, np.where(still, 0.0, 9e-4)]))
    host, dev = call(bits.edges_host, x, 2, n), call(bits.edges_device, x, 2, n)
    for k, name in enumerate(("general cross-section", "rectangular")):
        bad = differ(host[k], dev[k])
        assert not bad.any(), (name, bad.sum(), x[:, bad][:, :2], host[k][bad][:2], dev[k][bad][:2])


def test_published_words(bits):
    # the one pattern that marks an unpublished word is a NaN in both readings of a word (a double, a pair
    # of floats), and so is what stands for it; every other word passes unchanged
    w = np.array([0xFFFFFFFFFFFFFFFF, 0, 1, 0x3FF0000000000000, 0x7FF8000000000000, 0xFFFFFFFFFFFFFFFE], np.uint64)
    out = call(bits.publish_device, w, 1, w.size)[0]
    assert (out[1:] == w[1:]).all()
    assert out[0] != w[0]
    assert np.isnan(out[:1].view(np.float64)).all() and np.isnan(out[:1].view(np.float32)).all()
