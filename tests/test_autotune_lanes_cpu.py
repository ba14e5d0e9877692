"""The sub-step lanes that the launch-shape tuner tries (CPU, the stand-in of test_autotune_cpu.py)."""

import pytest

from wflow_gb300 import autotune
from test_autotune_cpu import StandIn, cost_of


@pytest.mark.parametrize("lanes", [0, 1, 2, 4, 8, 16])
def test_every_lane_count_can_win(lanes):
    def cost(t):
        c = cost_of(dict(t, substep_lanes=0, separate_overland_river=1))
        c["river"] -= 0.5 if t.get("substep_lanes", 0) == lanes else 0.0
        return c

    m = StandIn(cost)
    choice, results = autotune.tune(m, lambda s: (None, None, None))
    assert choice["substep_lanes"] == lanes
    assert (choice["routing_warps"], choice["routing_blocks_per_sm"]) == (4, 2)
