"""Exact-form states where the replaced division by six does not apply (derivative sums that
underflow, vanish or overflow) against the oracle's steps: the same bits."""
import numpy as np
import pytest

import ucb
from helpers import LORENZ, rk4_body
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("numb", ["f64", "f32"])
@pytest.mark.parametrize("lo,hi", [(0.0, 1.0), (0.0, 1e-18), (1e-21, 1e-17), (1e-40, 1e-44), (1e-287, 1e-290),
                                   (1e-300, 1e-306), (1e-310, 0.0), (1e12, 1e30), (1e100, 1e250)])
def test_exact_states_outside_the_normal_range(lo, hi, numb):
    """Lorenz with rho < 1 (everything decays to the origin) over initial x, y between lo and
    hi: from normal numbers through the threshold to subnormals, exact zeros, and blow-up."""
    n, steps, values = 7, 230, (0.0, 10.0, 0.5, 8 / 3)
    body = rk4_body(LORENZ)
    eng = ucb.Engine(0)
    req = ucb.Engine.lle2d_request(body, 3, (0.0, 0.0, lo), values, n_pts=n, sweep_over_var=True,
                                   sweep_over_var_2=True, var_sweep_index=0, var_sweep_index_2=1, param_lo=lo,
                                   param_hi=hi, param_lo_2=lo, param_hi_2=hi, h=0.01, t_max=1.0, NT=0.1, max_value=0.0,
                                   opt=ucb.options(precision=ucb.PREC_F32 if numb == "f32" else ucb.PREC_F64,
                                                   mode=ucb.MODE_EXACT))
    got = eng.lle2d_states(req, steps)
    eng.close()
    krs = O.Krs(body, 3, numb)
    ax = O.axis_values(n, lo, hi, numb=numb)
    want = np.empty((n * n, 3))
    for cell in range(n * n):
        x = np.array((ax[cell % n], ax[cell // n], lo), dtype=krs.dtype)
        want[cell] = krs.steps(x, np.array(values), 0.01, steps)
    np.testing.assert_array_equal(got, want)
    finite = np.isfinite(want)
    np.testing.assert_array_equal(np.signbit(got)[finite], np.signbit(want)[finite])
