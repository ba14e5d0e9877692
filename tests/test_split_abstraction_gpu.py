"""River abstractions (negative external inflow) in the split form over several sub-steps, fixed and
adaptive: against the FP64 oracle at the split form's bars."""

import pytest

from wflow_gb300 import abi, synthetic
from test_gpu_parity import split_errors

pytestmark = pytest.mark.gpu


def domain():
    dom = synthetic.make_domain(40, 500.0, seed=35, river_min_cells=6)
    ext = dom.river["river_external_inflow"]
    ext[::3] = -0.5
    ext[1::7] = 0.2
    return dom


@pytest.mark.parametrize("dt,adaptive", [(86400.0, False), (7200.0, False), (3600.0, True)])
def test_against_the_oracle(gpu_lib, dt, adaptive):
    w = split_errors(domain(), synthetic.make_config(dt, adaptive=adaptive, form=abi.WF_FORM_SPLIT), 4)
    assert w["outlet_q"] <= 1e-4, w
    assert w["soil_storage"] <= 1e-4, w
    assert w["closure"] <= 1e-7, w
