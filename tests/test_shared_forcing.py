"""Builds whose warp evaluates a forcing phase once for all its cells against the build that
evaluates it per cell: sweeping the phase over a range of width zero selects the latter for
the same trajectories."""
import numpy as np
import pytest

import ucb
from helpers import DUFFING, rk4_body

pytestmark = pytest.mark.gpu
PHASE, V = 0.7, 0.3


def options(prec):
    return ucb.options(precision=ucb.PREC_F32 if prec == "f32" else ucb.PREC_F64)


def axis(n, v, prec):
    """The engine's axis values over [v, v]: (1 - t) v + t v, an ulp off v at some t."""
    t = np.float32 if prec == "f32" else np.float64
    return np.array([t(v) if n == 1 else (t(1) - t(i) / t(n - 1)) * t(v) + t(i) / t(n - 1) * t(v) for i in range(n)])


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("n", [1, 5, 8, 13])
@pytest.mark.parametrize("transient,t_max,pre,maxv", [(0.0, 0.9, 1, 1e6), (6.2, 15.8, 1, 1e6), (31.7, 40.0, 3, 1e6),
                                                      (10.0, 25.0, 1, 2.6)])
def test_basin_features(prec, n, transient, t_max, pre, maxv):
    """Grids that leave lanes of the last warp without a cell, horizons around the table's
    and the divergence test's lengths, and a max_value that ends some cells early."""
    eng = ucb.Engine(0)
    got = []
    for y_var, lo2, hi2 in ((1, V, V), (2, PHASE, PHASE)):
        req = ucb.Engine.basins_dbscan_request(
            rk4_body(DUFFING), 3, (0.0, V, PHASE), (0.0,), n_pts=n, axis_x_var=0, axis_y_var=y_var, axis_x_lo=-2.5,
            axis_x_hi=2.6, axis_y_lo=lo2, axis_y_hi=hi2, h=2 * np.pi / 200, t_max=t_max, transient_time=transient,
            pre_scaller=pre, max_value=maxv, opt=options(prec))
        got.append(eng.run_basins_dbscan(req))
    eng.close()
    # the rows where both axes start the same trajectories
    t = np.float32 if prec == "f32" else np.float64
    rows = (axis(n, V, prec) == t(V)) & (axis(n, PHASE, prec) == t(PHASE))
    assert rows.sum() >= 0.7 * n
    for a, b in zip(got[0][:4], got[1][:4]):
        np.testing.assert_array_equal(a.reshape(n, n)[rows], b.reshape(n, n)[rows])
    if rows.all():
        assert got[0][4].steps == got[1][4].steps


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("writable", [0, 2, -1])
def test_diagram_of_a_state_sweep(prec, writable):
    """A diagram over initial x (the warp shares the phase) against single points that sweep
    the phase over one value; the phase itself and the combination with it recorded too."""
    eng = ucb.Engine(0)
    base = dict(writable_var=writable, h=2 * np.pi / 200, transient_time=9.0, t_max=60.0, max_peaks=40,
                opt=options(prec))
    xs = np.linspace(-1.5, 1.5, 7)
    kw = dict(sweep_over_var=True, n_pts=7, var_sweep_index=0, param_lo=-1.5, param_hi=1.5)
    counts, peaks, intervals, _ = eng.run_bif1d(
        ucb.Engine.bif1d_request(rk4_body(DUFFING), 3, (0.0, V, PHASE), (0.0,), **kw, **base))
    for i, x in enumerate(xs):
        t = np.float32 if prec == "f32" else np.float64
        x = (t(1.0) - t(i) / t(6)) * t(-1.5) + t(i) / t(6) * t(1.5)  # the axis value as the engine forms it
        kw = dict(sweep_over_var=True, n_pts=1, var_sweep_index=2, param_lo=PHASE, param_hi=PHASE)
        c, p, d, _ = eng.run_bif1d(
            ucb.Engine.bif1d_request(rk4_body(DUFFING), 3, (float(x), V, PHASE), (0.0,), **kw, **base))
        assert c[0] == counts[i]
        np.testing.assert_array_equal(p[0], peaks[i])
        np.testing.assert_array_equal(d[0], intervals[i])
    eng.close()
