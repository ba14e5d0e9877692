"""The split form's slim wavefronts at the sizes and settings where their launch changes: domains smaller
than a warp's work, chains alone in a warp or packed, members up to more than a warp, more sub-steps than
lanes and than a launch holds, cells with three and more upstream cells. Against the oracle at the split
form's bars (outlet discharge and soil storage 1e-4, water balance closure 1e-7), and over launch shapes,
which change the order of no sum within a sub-step: discharges stay the same bit for bit."""

import numpy as np
import pytest

from wflow_gb300 import abi, synthetic
from wflow_gb300.model import Model
from test_gpu_parity import split_errors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,ny,dt", [(5, 3, 3600.0), (17, 23, 86400.0), (97, 101, 3600.0), (41, 67, 86400.0)])
def test_sizes(gpu_lib, side, ny, dt):
    dom = synthetic.make_domain(side, 500.0, seed=41, ny=ny, river_min_cells=6)
    w = split_errors(dom, synthetic.make_config(dt, form=abi.WF_FORM_SPLIT), 4)
    assert w["outlet_q"] <= 1e-4, w
    assert w["soil_storage"] <= 1e-4, w
    assert w["closure"] <= 1e-7, w


@pytest.mark.parametrize("members", [1, 2, 32, 64])
@pytest.mark.parametrize("dt,river_dt", [(3600.0, 900.0), (86400.0, 900.0), (7200.0, 700.0)])
def test_launch_shapes(gpu_lib, members, dt, river_dt):
    dom = synthetic.make_domain(37, 500.0, seed=42, ny=29, river_min_cells=6)
    cfg = synthetic.make_config(dt, n_members=members, form=abi.WF_FORM_SPLIT)
    cfg.river_dt_fixed = river_dt
    models = [Model(cfg, dom) for _ in range(4)]
    for m, kw in zip(models[1:], (dict(substep_lanes=1), dict(substep_lanes=8, routing_warps=1),
                                  dict(routing_blocks_per_sm=1, routing_warps=8))):
        m.set_tuning(**kw)
    for s in range(2):
        P, PET, T = (np.tile(x, members) for x in synthetic.forcing(s, cfg.dt, dom.n_land, seed=42, precip_scale=3.0))
        for m in models:
            m.run_timestep(P, PET, T)
    for f in ["SSF_Q", "SATURATED_WATER_DEPTH", "LAND_Q", "RIVER_Q"]:
        want = models[0].get_value(f)
        for m in models[1:]:
            assert np.array_equal(m.get_value(f), want), f
    assert np.abs(models[0].get_value("RIVER_Q")).max() > 0.0
    for m in models:
        m.close()
