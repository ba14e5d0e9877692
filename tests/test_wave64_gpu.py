"""The FP64 form's slim wavefronts against the oracle at the sizes and settings where their launch
changes: chains alone in a warp or packed, more sub-steps than lanes and than a launch holds, sub-steps
of unequal size (launches are cut there), members up to more than a warp, cells with three and more
upstream cells, drained cells that get water again, and river cells with an abstraction. The bar is the
FP64 form's: relative 1e-9, at least 99.9 % of the values bit for bit."""

import numpy as np
import pytest

from wflow_gb300 import abi, synthetic
from wflow_gb300.model import Model
import oracle_py as O
from test_gpu_parity import LAND, RIVER, assert_parity, compare

pytestmark = pytest.mark.gpu


def run(dom, cfg, steps, members=1, wet=lambda s: 1.0, params=None):
    gpu, orc = Model(cfg, dom, params=params), O.OracleModel(cfg, dom, params=params)
    results = []
    for s in range(steps):
        P, PET, T = synthetic.forcing(s, cfg.dt, dom.n_land, seed=5)
        P = np.concatenate([P * wet(s) * (1.0 + 0.3 * m) for m in range(members)])
        PET, T = np.tile(PET, members), np.tile(T, members)
        gpu.run_timestep(P, PET, T)
        orc.set_forcing(P, PET, T)
        orc.step()
        results.append(compare(gpu, orc, LAND + RIVER, layers=gpu.N))
    gpu.close()
    assert_parity(results)


@pytest.mark.parametrize("side,ny", [(5, 3), (17, 23), (97, 101)])
@pytest.mark.parametrize("dt", [3600.0, 86400.0])
def test_sizes(gpu_lib, side, ny, dt):
    run(synthetic.make_domain(side, 500.0, seed=31, ny=ny, river_min_cells=6), synthetic.make_config(dt), 3)


@pytest.mark.parametrize("members", [2, 32, 64])
def test_members(gpu_lib, members):
    run(synthetic.make_domain(19, 500.0, seed=32, river_min_cells=6), synthetic.make_config(86400.0, n_members=members),
        2, members)


@pytest.mark.parametrize("land_dt,river_dt,ssf_dt", [(2500.0, 700.0, 86400.0), (120.0, 90.0, 1000.0)])
def test_unequal_and_many_substeps(gpu_lib, land_dt, river_dt, ssf_dt):
    cfg = synthetic.make_config(7200.0)
    cfg.land_dt_fixed, cfg.river_dt_fixed, cfg.subsurface_dt_fixed = land_dt, river_dt, ssf_dt
    run(synthetic.make_domain(24, 500.0, seed=33, river_min_cells=6), cfg, 3)


def test_drained_cells_get_water_again(gpu_lib):
    # rain for two days, three dry ones (rivers evaporate to the solve's floor), rain again
    run(synthetic.make_domain(48, 1000.0, seed=34), synthetic.make_config(86400.0), 7,
        wet=lambda s: 0.0 if 2 <= s < 5 else 2.0)


@pytest.mark.parametrize("dt,adaptive", [(86400.0, False), (900.0, False), (3600.0, True)])
def test_abstraction(gpu_lib, dt, adaptive):
    dom = synthetic.make_domain(40, 500.0, seed=35, river_min_cells=6)
    ext = dom.river["river_external_inflow"]
    ext[::3] = -0.5
    ext[1::7] = 0.2
    run(dom, synthetic.make_config(dt, adaptive=adaptive), 4)
