"""Linked reservoirs in a domain of many rivers, where the linked path's chain is joined by a longer
tributary near its head (tests/test_hinted_plan_cpu.py: such a chain has a chunk of its own): both forms
against the oracle at the bars of the linked reservoirs' other tests."""

import numpy as np
import pytest

from wflow_gb300 import abi, synthetic
from test_gpu_parity import assert_parity
from test_gpu_reservoirs import reservoir_closure, run_res_pair, split_res_errors

pytestmark = pytest.mark.gpu

LINK = 4  # river cells from the upper to the lower reservoir


def many_rivers(n=300):
    """n straight rivers of one length, which fill the group of chains with chunks of their own, and a
    small catchment, whose chains share a chunk."""
    parts = [synthetic.make_domain(40, 500.0, seed=500 + k, ny=1, river_min_cells=3) for k in range(n)]
    return synthetic.concat_domains(parts + [synthetic.make_domain(14, 500.0, seed=8, ny=9, river_min_cells=1)])


def low_link(dom):
    """An upper reservoir on a river's first cell, which joins a tributary several cells long, and a lower
    one LINK cells downstream; of make_linked_reservoirs' kinds."""
    rds = np.asarray(dom.river["river_downstream"])
    height = np.zeros(rds.size, int)
    for v in np.argsort(dom.upstream_cells[dom.river["river_land_index"]], kind="stable"):
        if rds[v] >= 0:
            height[rds[v]] = max(height[rds[v]], height[v] + 1)
    joined = np.zeros(rds.size, int)
    np.add.at(joined, rds[rds >= 0], 1)

    def below(v, k):
        while k and v >= 0:
            v, k = int(rds[v]), k - 1
        return v

    pairs = [(u, below(u, LINK)) for u in np.nonzero((height == 0) & (rds >= 0))[0]
             if joined[rds[u]] > 1 and height[rds[u]] >= 4 and below(u, LINK + 1) >= 0]
    up, lo = pairs[len(pairs) // 2]
    res = synthetic.make_linked_reservoirs(dom, seed=3)
    keep = [int(v) for v in res["river_index"][2:]]
    assert not {up, lo, int(rds[up]), int(rds[lo])} & (set(keep) | {int(rds[v]) for v in keep})
    res["river_index"] = np.array([up, lo, *keep], np.int32)
    return res


def test_fp64(gpu_lib):
    dom = many_rivers()
    gpu, orc, results, _ = run_res_pair(dom, low_link(dom), synthetic.make_config(86400.0), 4, check_every=2)
    assert_parity(results)
    assert np.array_equal(gpu.outlets(0), orc.outlets(0))
    assert reservoir_closure(gpu) <= 1e-9


def test_split(gpu_lib):
    dom = many_rivers()
    w = split_res_errors(dom, low_link(dom), synthetic.make_config(86400.0, form=abi.WF_FORM_SPLIT), 4)
    assert w["outlet_q"] <= 1e-4, w
    assert w["storage"] <= 1e-5, w
    assert w["outflow"] <= 1e-4, w
    assert w["res_closure"] <= 1e-9, w
