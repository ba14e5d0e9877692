"""The work a user has this framework do, as timed cases over its public entry points.

SBM cases: one pass is a stretch of model steps of a catchment that the program keeps in hand
(`Model`): the forcing of each step goes in from page-locked host memory, the outlet discharge comes
out every step, and the state maps a run writes out are read at the end of the pass. A pass goes on
from the state the last one left, over a cycle of forcing that holds wet, dry, warm and cold
stretches, as a running model does. The FP64 form is driven the way Wflow drives it (forcing, step,
read, one after the other), the split form the way an ensemble or forecast program does (FP32
forcing, the copy of the next step's forcing under the step that runs); its maps are kept in single
precision, as such a program writes them to file.

Local-inertial cases: one pass is an event on a river network or a land grid with its river, from a
warm state that the pass sets, over one or more hourly steps of runoff.

`exact` restates the local-inertial schemes in plain numpy. It gives None for the SBM cases: the
soil column and the three routing sweeps visit every cell of the drainage network in order, step by
step and sub-step by sub-step, which plain array code does not do within seconds, so those
outputs are held to the bounds of their types.
"""

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "wflow.jl_gb300"))

from wflow_gb300 import abi, synthetic  # noqa: E402
from wflow_gb300.li_river import LiDomain, LiRiver  # noqa: E402
from wflow_gb300.model import Model  # noqa: E402

DAY, HOUR = 86400.0, 3600.0

# Maps read at the end of a pass: what Wflow's example configurations write out (river and overland
# discharge, subsurface flow, soil water, evapotranspiration, total storage) and the states beside
# them (depths, snow, unsaturated store).
MAPS = ("RIVER_Q_AVERAGE", "LAND_Q_AVERAGE", "SSF_Q", "SATURATED_WATER_DEPTH", "ACTUAL_EVAPOTRANSPIRATION",
        "TOTAL_STORAGE", "RIVER_H", "LAND_H", "SNOW_STORAGE", "UNSATURATED_STORE_DEPTH")
# An ensemble keeps the discharge, the wetness and the storage of every member.
ENSEMBLE_MAPS = ("RIVER_Q_AVERAGE", "SATURATED_WATER_DEPTH", "TOTAL_STORAGE")


def _sbm(name, side, dt, steps, form, **more):
    case = dict(kind="sbm", side=side, cell=1000.0 if dt == DAY else 250.0, dt=dt, steps=steps, form=form, members=1,
                catchments=0, reservoirs=0, snow_transport=False, adaptive=False)
    case.update(more)
    if name:
        case["name"] = name
    return case


def _li(name, kind, size, steps):
    case = dict(kind=kind, size=size, steps=steps)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # a plot or a small test catchment coupled step by step (BMI): nothing but latency
        _sbm("fp64_daily_16", 16, DAY, 1, "fp64"),
        # the daily drop-in on a small catchment of 1 km cells
        _sbm("fp64_daily_64", 64, DAY, 5, "fp64"),
        # the drop-in for an hourly flood model of a mid-size catchment, a grid of odd size
        _sbm("fp64_hourly_301", 301, HOUR, 6, "fp64"),
        # a calibration ensemble in double precision
        _sbm("fp64_hourly_ensemble8_128", 128, HOUR, 6, "fp64", members=8),
        # a regulated daily catchment: reservoirs on the river
        _sbm("fp64_daily_reservoirs_160", 160, DAY, 3, "fp64", reservoirs=12),
        # an alpine daily catchment: snow moving downhill and glaciers
        _sbm("fp64_daily_snow_200", 200, DAY, 3, "fp64", snow_transport=True),
        # one large hourly domain in the split form, a day between maps
        _sbm("split_hourly_1024", 1024, HOUR, 24, "split"),
        # an hourly forecast ensemble
        _sbm("split_hourly_ensemble64_256", 256, HOUR, 24, "split", members=64),
        # a large domain of fine cells with Courant sub-steps
        _sbm("split_adaptive_1500", 1500, HOUR, 6, "split", adaptive=True, cell=100.0),
        # a batch of uneven independent catchments, daily steps
        _sbm("split_daily_ragged40", 450, DAY, 3, "split", catchments=40),
        # flood modelling: a river network alone, and a land grid with its river
        _li("li_river_6000", "li_river", 6000, 1),
        _li("li_domain_384", "li_domain", 384, 1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed ranges."""
    kind = rng.choice(("daily", "hourly", "ensemble", "reservoirs", "snow", "split", "split_ensemble", "adaptive",
                       "ragged", "li_river", "li_domain"))
    if kind == "daily":
        return _sbm(None, _log(rng, 8, 160), DAY, rng.randint(1, 5), "fp64")
    if kind == "hourly":
        return _sbm(None, _log(rng, 40, 301), HOUR, rng.randint(1, 6), "fp64")
    if kind == "ensemble":
        return _sbm(None, _log(rng, 32, 128), HOUR, rng.randint(1, 6), "fp64", members=rng.choice((2, 4, 8)))
    if kind == "reservoirs":
        return _sbm(None, _log(rng, 48, 160), DAY, rng.randint(1, 3), "fp64", reservoirs=rng.randint(3, 12))
    if kind == "snow":
        return _sbm(None, _log(rng, 24, 200), DAY, rng.randint(1, 3), "fp64", snow_transport=True)
    if kind == "split":
        return _sbm(None, _log(rng, 100, 1024), HOUR, rng.randint(2, 24), "split")
    if kind == "split_ensemble":
        return _sbm(None, _log(rng, 48, 256), HOUR, rng.randint(2, 24), "split",
                    members=rng.choice((2, 4, 8, 16, 32, 64)))
    if kind == "adaptive":
        return _sbm(None, _log(rng, 128, 1500), HOUR, rng.randint(1, 6), "split", adaptive=True, cell=100.0)
    if kind == "ragged":
        return _sbm(None, _log(rng, 60, 450), DAY, rng.randint(1, 3), "split", catchments=rng.randint(6, 40))
    if kind == "li_river":
        return _li(None, "li_river", _log(rng, 200, 6000), 1)
    return _li(None, "li_domain", _log(rng, 65, 384), 1)


# ------------------------------------------------------------------------------ SBM model ----

def _sides(case):
    """Sides of a batch's catchments: log-spaced areas up to the case's largest side."""
    k, top = case["catchments"], case["side"]
    return [max(4, int(round(top * 30.0 ** (-i / (k - 1.0))))) for i in range(k)] if k > 1 else [top]


def _cells(case):
    return sum(s * s for s in _sides(case)) if case["catchments"] else case["side"] ** 2


def _glacier_params(params, n, rng):
    return dict(params, glacier_fraction=np.where(rng.random(n) < 0.3, rng.uniform(0.05, 0.6, n), 0.0),
                glacier_temperature_threshold_melt=np.full(n, 273.15),
                glacier_degree_day_factor=rng.uniform(2e-3, 5e-3, n) / DAY,
                glacier_snow_to_ice_fraction=np.full(n, 0.002 / DAY),
                glacier_initial_store=rng.uniform(0.5, 6.0, n))


def _pinned(a, dtype):
    """A page-locked host array, its pages touched by the device once, as a program's forcing
    buffers are after its first steps."""
    t = torch.from_numpy(np.ascontiguousarray(a, dtype=dtype)).pin_memory()
    t.to("cuda")
    return t.numpy()


def _prepare_sbm(case, seed):
    rng = np.random.default_rng([seed, 2])
    # the catchment is the case's: its terrain and with it the number of river cells; its soils,
    # vegetation and weather are the seed's
    if case["catchments"]:
        dom = synthetic.concat_domains([synthetic.make_domain(s, case["cell"], seed=1000 + k)
                                        for k, s in enumerate(_sides(case))])
    else:
        dom = synthetic.make_domain(case["side"], case["cell"], seed=case["side"])
    dom.params = synthetic.make_params(dom.n_land, seed)
    n, members, dt, split = dom.n_land, case["members"], case["dt"], case["form"] == "split"
    cfg = synthetic.make_config(dt, n_members=members, form=abi.WF_FORM_SPLIT if split else abi.WF_FORM_FP64,
                                adaptive=case["adaptive"], per_member_soil=members > 1)
    params, pfac = dom.params, np.ones(members)
    if members > 1:
        kv0, f, pfac = synthetic.perturb_members(dom.params, members, seed=seed)
        params = dict(dom.params, kv_0=kv0, f=f)
    if case["adaptive"]:
        pfac = pfac * 3.0
    if case["snow_transport"]:
        cfg.snow_gravitational_transport = cfg.glacier = 1
        params = _glacier_params(params, n, rng)
    reservoirs = synthetic.make_reservoirs(dom, case["reservoirs"], seed=seed) if case["reservoirs"] else None
    model = Model(cfg, dom, params=params, reservoirs=reservoirs)
    # three steps of forcing, used in turn: an ordinary day or hour, a cold one and a dry one. An
    # ensemble perturbs the precipitation only; FP32 forcing takes the rest once for all members.
    dtype = np.float32 if split else np.float64
    forcing, at_reservoirs = [], []
    start = 230 if case["snow_transport"] else 0
    for s in range(3):
        P, PET, T = synthetic.forcing(start + s, dt, n, seed=seed)
        P = P * (1.0, 0.5, 0.0)[s]
        T = T + (0.0, -9.0, 3.0)[s]
        if reservoirs is not None:
            at_reservoirs.append(synthetic.reservoir_forcing(dom, reservoirs, P, PET, members))
        P = np.concatenate([P * x for x in pfac])
        if members > 1 and not split:
            PET, T = np.tile(PET, members), np.tile(T, members)
        forcing.append(tuple(_pinned(a, dtype) for a in (P, PET, T)))
    return dict(case=case, model=model, forcing=forcing, at_reservoirs=at_reservoirs, at=0)


def _run_sbm(state):
    case, model, forcing = state["case"], state["model"], state["forcing"]
    first, steps = state["at"], case["steps"]
    state["at"] = (first + steps) % len(forcing)
    split = case["form"] == "split"
    outlets = []
    if split and not case["adaptive"]:
        model.set_forcing_f32(*forcing[first % 3], asynchronous=True)
        for s in range(first, first + steps):
            model.step_async()
            if s + 1 < first + steps:
                model.set_forcing_f32(*forcing[(s + 1) % 3], asynchronous=True)
            outlets.append(model.outlets())
        model.synchronize()
    else:
        for s in range(first, first + steps):
            if state["at_reservoirs"]:
                rain, evaporation = state["at_reservoirs"][s % 3]
                model.set_value("RESERVOIR_PRECIPITATION", rain)
                model.set_value("RESERVOIR_EVAPORATION", evaporation)
            if split:
                model.set_forcing_f32(*forcing[s % 3])
                model.update_model()
            else:
                model.run_timestep(*forcing[s % 3])
            outlets.append(model.outlets())
    maps = ENSEMBLE_MAPS if case["members"] > 1 else MAPS
    out = {name: model.get_value(name) for name in maps}
    out["outlets"] = np.stack(outlets)
    if case["reservoirs"]:
        out["RESERVOIR_STORAGE"] = model.get_value("RESERVOIR_STORAGE")
        out["RESERVOIR_OUTFLOW_AVERAGE"] = model.get_value("RESERVOIR_OUTFLOW_AVERAGE")
    if case["snow_transport"]:
        out["SNOW_WATER"] = model.get_value("SNOW_WATER")
        out["GLACIER_STORE"] = model.get_value("GLACIER_STORE")
    return {k: v.astype(np.float32) for k, v in out.items()} if split else out


# Values per cell (the river: per river cell, about a fifth of the cells) that a step cannot do
# without: parameters, forcing, states read and written, fluxes and balance errors written. The
# split form's states and fluxes hold 48 bits in 8 bytes, its parameters and forcing 4 bytes.
_PARAMETERS, _FORCING, _STATES, _FLUXES = 50, 3, 14, 26
_RIVER_SHARE, _RIVER_PARAMETERS, _RIVER_STATES, _RIVER_FLUXES = 0.2, 6, 3, 8
_FLOPS_COLUMN, _FLOPS_WAVE = 600, 60  # soil column with its powers; one kinematic-wave solve


def _work_sbm(case):
    n, m, steps, dt = _cells(case), case["members"], case["steps"], case["dt"]
    p = 4 if case["form"] == "split" else 8
    land = n * (_PARAMETERS * p + m * (_FORCING * p + (2 * _STATES + _FLUXES) * 8))
    river = n * _RIVER_SHARE * (_RIVER_PARAMETERS * p + m * (2 * _RIVER_STATES + _RIVER_FLUXES) * 8)
    substeps = 1 + math.ceil(dt / HOUR) + _RIVER_SHARE * math.ceil(dt / 900.0)
    maps = len(ENSEMBLE_MAPS if m > 1 else MAPS)
    return {"bytes": steps * (land + river) + maps * n * m * 8,
            "flops": steps * n * m * (_FLOPS_COLUMN + substeps * _FLOPS_WAVE)}


# ------------------------------------------------------------------- local-inertial river ----

def _river_network(size, seed):
    """A river tree of `size` cells, each draining to one of the next forty, with four outlets of
    fixed depth; beds fall downstream, depths start wet, dry and about the threshold."""
    rng = np.random.default_rng([seed, 3])
    nb = 4
    n = size + nb
    i = np.arange(size)
    dst = np.minimum(i + 1 + rng.integers(0, 39, size), n - 1)
    dst[size - nb:] = size + np.arange(nb)
    length = rng.uniform(200.0, 1200.0, n)
    width = rng.uniform(5.0, 60.0, n)
    manning = rng.uniform(0.02, 0.05, n)
    zb = np.zeros(n)
    zb[size:] = rng.uniform(0.0, 2.0, nb)
    fall = length[:size] * rng.uniform(1e-5, 2e-3, size)
    for k in range(size - 1, -1, -1):
        zb[k] = zb[dst[k]] + fall[k]
    h = rng.uniform(0.0, 3.0, n)
    sort = rng.integers(0, 10, n)
    h[sort == 0] = 0.0
    h[sort == 1] = 1e-3 * rng.uniform(0.5, 1.5, int((sort == 1).sum()))
    n_e = (manning[dst] * length[dst] + manning[:size] * length[:size]) / (length[dst] + length[:size])
    external = np.zeros(n)
    external[rng.choice(size, max(2, size // 50), replace=False)] = rng.uniform(0.0, 10.0, max(2, size // 50))
    return dict(n_active=size, src=i, dst=dst, zb=zb, flow_length=length, flow_width=width, h=h,
                zb_edge=np.maximum(zb[:size], zb[dst]), width_edge=np.minimum(width[dst], width[:size]),
                length_edge=0.5 * (length[dst] + length[:size]), mannings_n_sq_edge=n_e * n_e,
                inwater=rng.uniform(0.0, 5.0, n) * (rng.random(n) < 0.7), external_inflow=external)


def _prepare_river(case, seed):
    r = _river_network(case["size"], seed)
    net = {k: r[k] for k in ("src", "dst", "zb", "flow_length", "flow_width", "zb_edge", "width_edge", "length_edge",
                             "mannings_n_sq_edge", "n_active")}
    model = LiRiver(h_init=r["h"], **net)
    model.set_boundary(external_inflow=r["external_inflow"])
    return dict(case=case, model=model, net=r, q=np.zeros(case["size"]))


def _run_river(state):
    model, net = state["model"], state["net"]
    model.set_state(net["h"], state["q"])
    model.set_inwater(net["inwater"])
    for _ in range(state["case"]["steps"]):
        model.step(HOUR)
    return {k: model.get(k) for k in ("h", "storage", "q", "q_average")}


# ------------------------------------------------- local-inertial land grid with its river ----

def _li_grid(case, seed):
    return synthetic.li_grid(case["size"], case["size"], seed=seed, river_every=min(64, case["size"] // 2))


def _prepare_domain(case, seed):
    land, river, h_river, h_land, runoff = _li_grid(case, seed)
    return dict(case=case, model=LiDomain(land, river, h_river), h_land=h_land, h_river=h_river, runoff=runoff,
                still=np.zeros(len(h_land)), still_river=np.zeros(len(river["src"])))


def _run_domain(state):
    model = state["model"]
    model.set_state(state["h_land"], state["h_river"], state["still"], state["still"], state["still_river"])
    model.set_inputs(state["runoff"])
    for _ in range(state["case"]["steps"]):
        model.step(HOUR)
    return {k: model.get(k) for k in ("h_land", "qx_average", "qy_average", "h_river", "q_river_average")}


def _work_li(case):
    # per cell of the pass: geometry and elevations, state in and out, cumulative fluxes; per
    # sub-step (an hour of 100 m cells a metre or two deep takes about 250) the flux and depth updates
    land = case["kind"] == "li_domain"
    n = case["size"] ** 2 if land else case["size"]
    return {"bytes": n * ((14 + 2 * 4 + 5) if land else (10 + 2 * 3 + 4)) * 8.0,
            "flops": case["steps"] * 250.0 * n * (2 * 30 + 12 if land else 42)}


# ------------------------------------------------------- plain numpy, double precision ----
# The schemes of Wflow's local-inertial routing (Wflow/src/routing/surface/
# surface_process.jl:88-163, surface_staggered_scheme.jl).

_G = 9.80665


def _edge_flow(net, h, q, dt):
    """Discharge of every river edge after a sub-step."""
    a, b = net["src"], net["dst"]
    z0, z1 = net["zb"][a] + h[a], net["zb"][b] + h[b]
    hf = np.maximum(z0, z1) - net["zb_edge"]
    wet = hf > 1e-3
    depth = np.where(wet, hf, 1.0)
    area = net["width_edge"] * depth
    radius = area / (2.0 * depth + net["width_edge"])
    slope = (z1 - z0) / net["length_edge"]
    new = (q - _G * area * dt * slope) / (
        1.0 + _G * dt * net["mannings_n_sq_edge"] * np.abs(q) / (np.cbrt(radius ** 4) * area))
    critical = np.sqrt(_G * depth) * area
    new = np.where(np.abs(new) > critical, np.sign(new) * critical, new)
    new = np.where(wet, new, 0.0)
    new = np.where(h[a] <= 0.0, np.minimum(new, 0.0), new)
    return np.where(h[b] <= 0.0, np.maximum(new, 0.0), new)


def _exact_river(case, seed):
    net = _river_network(case["size"], seed)
    n, na = len(net["zb"]), case["size"]
    h = net["h"].copy()
    plan = net["flow_length"] * net["flow_width"]
    storage = np.concatenate([(h * plan)[:na], np.zeros(n - na)])
    q, total = np.zeros(na), np.zeros(na)
    for _ in range(case["steps"]):
        t, total = 0.0, np.zeros(na)
        while t < HOUR:
            with np.errstate(divide="ignore"):
                dt = np.min(0.7 * net["flow_length"] / np.sqrt(_G * h))
            dt = 60.0 if np.isinf(dt) else dt
            dt = HOUR - t if t + dt > HOUR else dt
            q = _edge_flow(net, h, q, dt)
            total += q * dt
            into, out = (np.bincount(net[k], weights=q, minlength=n)[:na] for k in ("dst", "src"))
            storage[:na] = np.maximum(storage[:na] + (into - out + net["inwater"][:na]) * dt, 0.0)
            storage[:na] += net["external_inflow"][:na] * dt
            h[:na] = storage[:na] / plan[:na]
            t += dt
    return {"h": h, "storage": storage, "q": q, "q_average": total / HOUR}


def _land_flow(land, h, q, dt, x_dir):
    """Discharge of every land edge of one direction after a sub-step."""
    n = len(h)
    u, d = (land["ind_x_up"], land["ind_x_down"]) if x_dir else (land["ind_y_up"], land["ind_y_down"])
    width = land["ywidth_at_edge"] if x_dir else land["xwidth_at_edge"]
    length = land["x_length"] if x_dir else land["y_length"]
    there = (u < n) & (width != 0.0)
    v = np.minimum(u, n - 1)
    z = land["elevation"]
    z0, z1 = z + h, z[v] + h[v]
    hf = np.maximum(z0, z1) - np.maximum(z, z[v])
    wet = there & (hf > 1e-3)
    depth, w = np.where(wet, hf, 1.0), np.where(there, width, 1.0)
    padded = np.append(q, 0.0)
    slope = (z1 - z0) / (0.5 * (length + length[v]))
    theta = land["theta"]
    new = (theta * q + 0.5 * (1.0 - theta) * (padded[u] + padded[d]) - _G * depth * w * dt * slope) / (
        1.0 + _G * dt * land["mannings_n_sq"] * np.abs(q) / (np.cbrt(depth ** 7) * w))
    critical = depth * np.sqrt(_G * depth) * w
    new = np.where(np.abs(new) > critical, np.sign(new) * critical, new)
    new = np.where(h <= 0.0, np.minimum(new, 0.0), new)
    new = np.where(h[v] <= 0.0, np.maximum(new, 0.0), new)
    return np.where(there, np.where(wet, new, 0.0), q), there


def _exact_domain(case, seed):
    land, river, h_river, h_land, runoff = _li_grid(case, seed)
    n, na, nr = len(h_land), river["n_active"], len(h_river)
    cells = np.empty(na, np.int64)
    at_river = land["river_index"] >= 0
    cells[land["river_index"][at_river]] = np.nonzero(at_river)[0]
    plan, plan_r = land["x_length"] * land["y_length"], river["flow_length"] * river["flow_width"]
    full_depth = river["bankfull_depth"][:na]
    full = full_depth * plan_r[:na]
    h, hr = h_land.copy(), h_river.copy()
    storage = h * plan
    storage[cells] = np.where(h[cells] > 0.0, full + storage[cells], hr[:na] * plan_r[:na])
    qx, qy, qr = np.zeros(n), np.zeros(n), np.zeros(len(river["src"]))
    xd, yd = land["ind_x_down"], land["ind_y_down"]
    for _ in range(case["steps"]):
        t, sx, sy, sr = 0.0, np.zeros(n), np.zeros(n), np.zeros(len(qr))
        while t < HOUR:
            with np.errstate(divide="ignore"):
                dt_r = np.min(river["alpha"] * river["flow_length"][:na] / np.sqrt(_G * hr[:na]))
                dt_l = np.min(np.where(at_river, np.inf, land["alpha"] * np.minimum(land["x_length"], land["y_length"])
                                       / np.sqrt(_G * h)))
            dt = min(60.0 if np.isinf(dt_r) else dt_r, 60.0 if np.isinf(dt_l) else dt_l)
            dt = HOUR - t if t + dt > HOUR else dt
            (qx, on_x), (qy, on_y) = _land_flow(land, h, qx, dt, True), _land_flow(land, h, qy, dt, False)
            sx += np.where(on_x, qx * dt, 0.0)
            sy += np.where(on_y, qy * dt, 0.0)
            qr = _edge_flow(river, hr, qr, dt)
            sr += qr * dt
            px, py = np.append(qx, 0.0), np.append(qy, 0.0)
            net = px[xd] - qx + py[yd] - qy + runoff
            into, out = (np.bincount(river[k], weights=qr, minlength=nr)[:na] for k in ("dst", "src"))
            net[cells] += into - out
            storage = np.maximum(storage + net * dt, 0.0)
            h = storage / plan
            s = storage[cells]
            spilled = s >= full
            hr[:na] = np.where(spilled, full_depth + (s - full) / plan[cells], s / plan_r[:na])
            h[cells] = np.where(spilled, hr[:na] - full_depth, 0.0)
            t += dt
    return {"h_land": h, "qx_average": sx / HOUR, "qy_average": sy / HOUR, "h_river": hr, "q_river_average": sr / HOUR}


# --------------------------------------------------------------------------------- by kind ----

_PREPARE = {"sbm": _prepare_sbm, "li_river": _prepare_river, "li_domain": _prepare_domain}
_RUN = {"sbm": _run_sbm, "li_river": _run_river, "li_domain": _run_domain}
_EXACT = {"li_river": _exact_river, "li_domain": _exact_domain}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["case"]["kind"]](state)


def work(case):
    return _work_sbm(case) if case["kind"] == "sbm" else _work_li(case)


def exact(case, seed):
    return _EXACT[case["kind"]](case, seed) if case["kind"] in _EXACT else None
