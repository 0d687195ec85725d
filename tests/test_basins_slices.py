"""Stroboscopic basins of maps that are taken in slices of periods (more cells than a warp a
scheduler) against the oracle, cell for cell: class, period and number of periods."""
import numpy as np
import pytest

import ucb
from helpers import LORENZ, rk4_body
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [137, 138, 160])
@pytest.mark.parametrize("cap", [63, 64, 65, 128, 130, 519])
def test_sliced_maps_match_oracle(n, cap):
    """Lorenz at rho = 10 (polynomial, so the exact form has the oracle's bits): cells settle on
    one of two fixed points after 40 to several hundred periods or leave through max_value, in
    slices of 1 to 65 periods; 137^2 cells are the largest map of one slice."""
    b = dict(n_pts=n, axis_x_var=0, axis_y_var=1, axis_x_lo=-40.0, axis_x_hi=40.0, axis_y_lo=-40.0, axis_y_hi=40.0,
             ic=(0.0, 0.0, 25.0), values=(0, 10.0, 10.0, 8 / 3), period=0.25, steps_per_period=25, max_periods=cap,
             match_count=20, match_tol=1e-6, phase_var=-1, max_value=100.0)
    eng = ucb.Engine(0)
    req = ucb.Engine.basins_request(rk4_body(LORENZ), 3, b["ic"], b["values"], n_pts=n, axis_x_lo=-40.0, axis_x_hi=40.0,
                                    axis_y_lo=-40.0, axis_y_hi=40.0, period=0.25, steps_per_period=25, max_periods=cap,
                                    match_count=20, match_tol=1e-6, max_value=100.0,
                                    opt=ucb.options(precision=ucb.PREC_F64, mode=ucb.MODE_EXACT))
    labels, periods, iters, att, res = eng.run_basins(req)
    eng.close()
    cells = np.sort(np.random.default_rng(cap).choice(n * n, 3000, replace=False))
    per, cx, cy, it = O.basins(O.Krs(rk4_body(LORENZ), 3), b, cells=cells)
    np.testing.assert_array_equal(periods[cells], per)
    np.testing.assert_array_equal(iters[cells], it)
    assert ((labels[cells] > 0) == (per > 0)).all() and ((labels[cells] < 0) == (per < 0)).all()
    for cell, p, x, y in zip(cells, per, cx, cy):
        if p > 0:
            a = att[labels[cell] - 1]
            assert a[0] == p and abs(a[1] - x) <= 1e-3 and abs(a[2] - y) <= 1e-3
    assert res.steps == 25 * int(iters.astype(np.int64).sum())
