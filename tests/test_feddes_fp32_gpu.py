"""The root water uptake reduction that an FP32 estimate of the soil-water head decides (FP64 form),
where FP32 says little: a porosity range theta_s - theta_r that is small against theta_s, and
parameters without a value. Against the oracle, relative 1e-9."""

import numpy as np
import pytest

from wflow_gb300 import synthetic
from test_gpu_parity import assert_parity, run_pair

pytestmark = pytest.mark.gpu


def soil(dom, seed):
    """The heads of the reduction (h3, h4) brought close to the soil's, so that many layers lie near them."""
    p = dict(dom.params)
    rng = np.random.default_rng([seed, 3])
    n = dom.n_land
    p["h3_high"] = p["h3_low"] = -(10.0 ** rng.uniform(-0.9, 0.5, n))
    p["h4"] = p["h3_high"] * (1.0 + rng.uniform(0.01, 0.3, n))
    return p, rng


@pytest.mark.parametrize("decades", [(-3.0, -2.0), (-5.0, -3.0), (-7.0, -5.0)])
def test_small_porosity_range(gpu_lib, decades):
    dom = synthetic.make_domain(48, 1000.0, seed=61)
    p, rng = soil(dom, 61)
    p["theta_r"] = p["theta_s"] - 10.0 ** rng.uniform(*decades, dom.n_land)
    _, _, res = run_pair(dom, synthetic.make_config(86400.0), 6, params=p)
    assert_parity(res)


def test_air_entry_pressure_without_a_value(gpu_lib):
    # NaN of either sign (a quotient 0 / 0 gives a negative one on x86)
    dom = synthetic.make_domain(24, 1000.0, seed=62)
    p, rng = soil(dom, 62)
    psi = p["air_entry_pressure"] = p["air_entry_pressure"].copy()
    some = rng.random(dom.n_land) < 0.2
    psi[some] = np.where(rng.random(some.sum()) < 0.5, 1.0, -1.0) * np.nan
    psi[some] = np.copysign(psi[some], np.where(rng.random(some.sum()) < 0.5, 1.0, -1.0))
    assert np.signbit(psi[some]).any()
    _, _, res = run_pair(dom, synthetic.make_config(86400.0), 4, params=p)
    assert_parity(res)
