"""Device memory of a model: no more than the bytes that the same model took when its sweeps carried no
terms and vectors of their own (a model near the memory limit still fits), and the sweeps' terms in
fields that the step writes later: the river's on a layout larger than the land's, where they do not fit."""

import numpy as np
import pytest

from wflow_gb300 import abi, synthetic
from wflow_gb300.model import Model
from test_gpu_parity import assert_parity
from test_gpu_reservoirs import reservoir_closure, run_res_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,members,side,limit", [
    (abi.WF_FORM_FP64, 1, 600, 713031680), (abi.WF_FORM_FP64, 8, 200, 364904448),
    (abi.WF_FORM_SPLIT, 1, 600, 987758592), (abi.WF_FORM_SPLIT, 64, 120, 784334848)])
def test_bytes_of_a_model(gpu_lib, form, members, side, limit):
    import gc
    import torch
    gc.collect()
    Model(synthetic.make_config(86400.0, form=form), synthetic.make_domain(8, 1000.0, seed=81)).close()  # module loads
    dom = synthetic.make_domain(side, 1000.0, seed=81)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    m = Model(synthetic.make_config(86400.0, form=form, n_members=members), dom)
    torch.cuda.synchronize()
    used = free - torch.cuda.mem_get_info()[0]
    m.close()
    assert 0 < used <= limit, used


def test_river_layout_larger_than_the_lands(gpu_lib):
    # every cell a river cell; the linked reservoirs' path changes the river's chains and their padding
    dom = synthetic.make_domain(48, 1000.0, seed=7, river_min_cells=0)
    res = synthetic.make_linked_reservoirs(dom, seed=3)
    gpu, orc, results, _ = run_res_pair(dom, res, synthetic.make_config(86400.0), 4, check_every=2)
    assert_parity(results)
    assert np.array_equal(gpu.outlets(0), orc.outlets(0))
    assert reservoir_closure(gpu) <= 1e-9
