"""The state that a sliced stroboscopic map keeps between its launches goes back to the device when
it is large: the engine's pool does not hold it after the call."""
import numpy as np
import pytest

import ucb
from helpers import DUFFING, rk4_body

pytestmark = pytest.mark.gpu


def test_large_state_is_given_back():
    import torch

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    def request(n, cap):
        return ucb.Engine.basins_request(rk4_body(DUFFING), 3, (0.0, 0.0, 0.0), (0.0,), n_pts=n, axis_x_lo=-2.5,
                                         axis_x_hi=2.5, axis_y_lo=-2.5, axis_y_hi=2.5, period=2 * np.pi,
                                         steps_per_period=20, max_periods=cap, phase_var=2, match_count=20,
                                         max_value=1e6, opt=ucb.options(precision=ucb.PREC_F64))

    eng = ucb.Engine(0)
    n = 2048  # 4.2 M cells: 50 MB of results, 770 MB of state
    eng.run_basins(request(n, 60))  # one launch (at most 64 periods): the results' buffers alone
    before, launched = free(), eng.launches
    eng.run_basins(request(n, 66))
    launched = eng.launches - launched
    assert launched == 3  # two slices and the labels
    assert before - free() < 64 << 20
    eng.close()
