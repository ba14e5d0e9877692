"""The device sub-step loops of the local-inertial schemes at the sizes where their launch shape
changes (blocks of 32 to 256 threads, a last block that is nearly empty, more cells than threads), and
with every cell at the same depth, where every cell is the smallest stable sub-step's: against the
oracle at the component's bar, relative 1e-9 and equal sub-step counts."""

import numpy as np
import pytest

from li_cases import OracleLi, OracleLiDomain, random_land_domain, random_river
from test_local_inertial_gpu import DOMAIN_FIELDS, _assert_same, _domain, _max_rel, _river

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_active", [5, 33, 4861, 9730, 41000])
def test_river_sizes(gpu_lib, n_active):
    net = random_river(21, n_active=n_active, n_bound=2)
    gpu, orc = _river(net), OracleLi(net)
    for m in (gpu, orc):
        m.set_state(net["h"])
        m.set_inwater(net["inwater"])
    assert gpu.step(900.0) == orc.step(900.0)
    _assert_same(gpu, orc, n_active)
    gpu.close()


def test_river_of_equal_depths(gpu_lib):
    net = random_river(22, n_active=5000, n_bound=2)
    net = dict(net, h=np.full(net["n"], 1.25), flow_length=np.full(net["n"], 500.0))
    gpu, orc = _river(net), OracleLi(net)
    for m in (gpu, orc):
        m.set_state(net["h"])
        m.set_inwater(net["inwater"])
    assert gpu.step(600.0) == orc.step(600.0)
    _assert_same(gpu, orc, "equal depths")
    gpu.close()


@pytest.mark.parametrize("nx,ny", [(9, 8), (33, 31), (150, 131)])
def test_domain_sizes(gpu_lib, nx, ny):
    land, river, h_river, state, inputs = random_land_domain(23, nx=nx, ny=ny)
    gpu, orc = _domain(land, river, h_river), OracleLiDomain(land, river, h_river)
    for m in (gpu, orc):
        m.set_state(**state)
        m.set_inputs(**inputs)
    assert gpu.step(600.0) == orc.step(600.0)
    for f in DOMAIN_FIELDS:
        assert _max_rel(gpu.get(f), orc.get(f)) <= 1e-9, f
    gpu.close()
