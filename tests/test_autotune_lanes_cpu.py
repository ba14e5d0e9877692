"""The launch-shape tuner on a model without variants of its sweeps, and the sub-step lanes it tries (CPU,
the stand-in of test_autotune_cpu.py)."""

import pytest

from wflow_gb300 import autotune
from wflow_gb300.model import Model
from test_autotune_cpu import StandIn, cost_of


class Plain(StandIn):
    SWEEP_VARIANTS = Model.SWEEP_VARIANTS


@pytest.mark.parametrize("lanes", [0, 1, 2, 4, 8, 16])
def test_every_lane_count_can_win(lanes):
    def cost(t):
        c = cost_of(dict(t, substep_lanes=0, separate_overland_river=1))
        c["river"] -= 0.5 if t.get("substep_lanes", 0) == lanes else 0.0
        return c

    m = Plain(cost)
    choice, results = autotune.tune(m, lambda s: (None, None, None))
    assert choice["substep_lanes"] == lanes
    assert (choice["routing_warps"], choice["routing_blocks_per_sm"]) == (4, 2)


def test_switches_without_effect_are_not_timed():
    seen = []
    m = Plain(cost_of)
    set_tuning = m.set_tuning
    m.set_tuning = lambda **kw: (seen.append(kw), set_tuning(**kw))
    choice, results = autotune.tune(m, lambda s: (None, None, None))
    assert not any(kw.get("sweep_inputs") for kw in seen)
    assert {r[0] for r in results} == {"routing", "lanes", "vertical"}
