"""River cells whose inflow, previous discharge and lateral inflow cancel exactly: the reference's zero
case (discharge and flow area 0, surface_process.jl:29-31), in the FP64 form against the oracle."""

import numpy as np
import pytest

from wflow_gb300 import abi, synthetic
from wflow_gb300.model import Model
import oracle_py as O
from test_gpu_parity import RIVER, assert_parity, compare

pytestmark = pytest.mark.gpu

F = abi.FIELD


def domain(seed=71):
    return synthetic.make_domain(9, 500.0, seed=seed, river_min_cells=3)


def heads(dom):
    """River cells without an upstream river cell."""
    rds = np.asarray(dom.river["river_downstream"])
    return np.setdiff1d(np.arange(rds.size), rds[rds >= 0])


def set_river(model, q, h, storage):
    for name, v in (("RIVER_Q", q), ("RIVER_H", h), ("RIVER_STORAGE", storage)):
        if isinstance(model, Model):
            model.set_value(name, v)
        else:
            model.set(F[name], v)


def test_abstraction_after_a_zero_sum(gpu_lib):
    # heads start with a stored volume, no discharge, and an abstraction equal to their lateral inflow:
    # the first sub-step is the zero case, which empties the cell, so the next one has nothing to
    # abstract from
    dom = domain()
    cfg = synthetic.make_config(3600.0)  # four river sub-steps
    P, PET, T = synthetic.forcing(0, cfg.dt, dom.n_land, seed=71, precip_scale=5.0)
    P = P + 2e-6
    river = dom.river
    first = heads(dom)
    q = np.full(dom.n_river, 0.1)
    q[first] = 0.0
    h = np.full(dom.n_river, 0.5)
    storage = h * river["river_width"] * river["river_length"]

    def oracle():
        m = O.OracleModel(cfg, dom)
        set_river(m, q, h, storage)
        m.set_forcing(P, PET, T)
        m.step()
        return m

    inwater = oracle().get(F["RIVER_INWATER"])
    assert (inwater[first] > 0.0).all()
    assert (0.8 * storage[first] / 900.0 > inwater[first]).all()
    river["river_external_inflow"][first] = -inwater[first]
    orc = oracle()
    assert (orc.get(F["RIVER_INWATER"]) == inwater).all()
    gpu = Model(cfg, dom)
    set_river(gpu, q, h, storage)
    gpu.run_timestep(P, PET, T)
    assert_parity([compare(gpu, orc, RIVER)])
    assert (orc.get(F["RIVER_Q"])[first] > 0.0).all()
    gpu.close()


def test_lateral_inflow_within_the_rounding_of_the_discharges(gpu_lib):
    # a negative previous discharge that cancels the inflow but for a rest of 2^-25 of them, which the
    # lateral inflow cancels
    dom = domain(72)
    cfg = synthetic.make_config(3600.0)
    cfg.river_dt_fixed = 3600.0  # one sub-step
    P, PET, T = synthetic.forcing(0, cfg.dt, dom.n_land, seed=72, precip_scale=5.0)
    river = dom.river
    rds = np.asarray(river["river_downstream"])
    n_up = np.bincount(rds[rds >= 0], minlength=rds.size)
    up = np.array([u for u in heads(dom) if rds[u] >= 0 and n_up[rds[u]] == 1])
    cells = rds[up]
    assert cells.size > 0
    q = np.full(rds.size, 3.0)
    h = np.full(rds.size, 0.5)
    storage = h * river["river_width"] * river["river_length"]

    def oracle():
        m = O.OracleModel(cfg, dom)
        set_river(m, q, h, storage)
        m.set_forcing(P, PET, T)
        m.step()
        return m

    # scale: the inflows must be large against the lateral inflow of the cells
    q[up] = 2.0e5
    orc = oracle()
    q_up, lateral = orc.get(F["RIVER_Q"])[up], orc.get(F["RIVER_INWATER"])[cells] / river["river_length"][cells]
    for c, qu, lat in zip(cells, q_up, lateral):
        rest = 2.0 ** np.ceil(np.log2(qu * 2.0 ** -25))
        assert lat < rest and qu > 0.0
        length = river["river_length"][c]
        ext = (rest - lat) * length  # lateral plus external inflow per length: exactly `rest`
        near = [e for k in range(-8, 9) if lat + (e := ext + k * np.spacing(ext)) / length == rest]
        assert near, c
        river["river_external_inflow"][c] = near[0]
        q[c] = -(qu + rest)
        assert qu + q[c] + rest == 0.0
    orc = oracle()
    assert (orc.get(F["RIVER_Q"])[cells] == 0.0).all()
    gpu = Model(cfg, dom)
    set_river(gpu, q, h, storage)
    gpu.run_timestep(P, PET, T)
    assert_parity([compare(gpu, orc, RIVER)])
    gpu.close()
