"""Every sweep takes the routing warps that set_tuning accepts: snow transport, subsurface sub-steps and
adaptive sub-steps run with 8 and 32 warps per block asked for, with the results of the default."""

import numpy as np
import pytest

from wflow_gb300 import abi, synthetic
from wflow_gb300.model import Model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warps", [8, 32])
@pytest.mark.parametrize("form", [abi.WF_FORM_FP64, abi.WF_FORM_SPLIT])
@pytest.mark.parametrize("kind", ["snow transport", "subsurface sub-steps", "adaptive"])
def test_many_routing_warps(gpu_lib, kind, form, warps):
    dom = synthetic.make_domain(20, 1000.0, seed=51)
    cfg = synthetic.make_config(86400.0, form=form, adaptive=kind == "adaptive")
    if kind == "snow transport":
        cfg.snow_gravitational_transport = 1
    if kind == "subsurface sub-steps":
        cfg.subsurface_dt_fixed = 20000.0
    a, b = Model(cfg, dom), Model(cfg, dom)
    b.set_tuning(routing_warps=warps)
    for s in range(3):
        P, PET, T = synthetic.forcing(230 + s, cfg.dt, dom.n_land, seed=51)
        for m in (a, b):
            m.run_timestep(P, PET, T - 8.0)
    for f in ["SNOW_STORAGE", "SSF_Q", "LAND_Q", "RIVER_Q", "TOTAL_SOIL_WATER_STORAGE"]:
        assert np.array_equal(a.get_value(f), b.get_value(f)), f
    a.close()
    b.close()
