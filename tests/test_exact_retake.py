"""Exact-form calls some of whose cells leave the range of the replaced division by six (their
derivative sums underflow while they settle on the origin): every path that takes blocks of steps
again gives the bits of the same body taken verbatim, and a warp takes one pass, not two. A body
whose division is spelled "/ 6 ;" is the same arithmetic and is not replaced."""
import numpy as np
import pytest

import ucb
from helpers import LORENZ, rk4_body

pytestmark = pytest.mark.gpu
BODY = rk4_body(LORENZ)
VERBATIM = BODY.replace(" / 6;", " / 6 ;")
VALUES = (0.0, 10.0, 0.5, 8 / 3)


@pytest.fixture(scope="module")
def eng():
    e = ucb.Engine(0)
    yield e
    e.close()


def options(prec, **kw):
    return ucb.options(precision=ucb.PREC_F32 if prec == "f32" else ucb.PREC_F64, mode=ucb.MODE_EXACT, **kw)


def sweep(n, prec, **kw):
    """rho from 0.2 (settles) to 28 (grows to the attractor)."""
    return dict(dict(n_pts=n, param_index=2, param_lo=0.2, param_hi=28.0, h=0.01, transient_time=1.3, max_value=1e6,
                     opt=options(prec)), **kw)


def plane(n, prec, **kw):
    return sweep(n, prec, **dict(dict(param_index_2=1, param_lo_2=5.0, param_hi_2=15.0), **kw))


def tiny(prec, scale):
    """A start from which the sums of settling cells cross the range's end within a few hundred steps
    (scale 1), or lie beyond it (1e-3), or vanish (0)."""
    x = (1e-17 if prec == "f32" else 1e-287) * scale
    return (x, x, x)


def both(run, request):
    out = []
    for body in (BODY, VERBATIM):
        got = run(request(body))
        out.append([np.asarray(v) for v in got[:-1]] + [got[-1].steps])
    assert len(out[0]) == len(out[1])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    return out[0]


def test_the_two_bodies_differ_in_spelling_only():
    assert BODY != VERBATIM and BODY.replace(" ", "") == VERBATIM.replace(" ", "")


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("scale", [1.0, 1e-3, 0.0])
@pytest.mark.parametrize("n", [40, 140])  # a trajectory a lane; pairs
@pytest.mark.parametrize("NT,nominal", [(0.1, False), (1.57, True)])
@pytest.mark.parametrize("eps", ["small", "large"])
def test_exponent_maps(eng, prec, scale, n, NT, nominal, eps):
    e = 1e-4 if eps == "large" else 1e-20 if prec == "f32" else 1e-290
    both(eng.run_lle2d, lambda body: ucb.Engine.lle2d_request(
        body, 3, tiny(prec, scale), VALUES, NT=NT, eps=e, t_max=9.5,
        **plane(n, prec, opt=options(prec, nominal_steps=nominal, lle_method=ucb.LLE_SHADOW))))


@pytest.mark.parametrize("prec,n", [("f64", 7), ("f64", 160), ("f32", 7), ("f32", 200)])  # groups; a cell a lane
@pytest.mark.parametrize("scale", [1.0, 1e-3])
@pytest.mark.parametrize("NT", [0.1, 1.57])
def test_spectra(eng, prec, n, scale, NT):
    both(eng.run_ls2d, lambda body: ucb.Engine.ls2d_request(
        body, 3, tiny(prec, scale), VALUES, method=ucb.LS_FIXED, NT=NT, eps=1e-6, t_max=8.0, **plane(n, prec)))


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("scale", [1.0, 1e-3])
@pytest.mark.parametrize("block", [0, 128])  # two warps for 32 points; one
@pytest.mark.parametrize("pre", [1, 3])
def test_diagrams(eng, prec, scale, block, pre):
    both(eng.run_bif1d, lambda body: ucb.Engine.bif1d_request(
        body, 3, tiny(prec, scale), VALUES, max_peaks=40, pre_scaller=pre, t_max=30.0,
        **sweep(100, prec, opt=options(prec, block_threads=block))))


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("scale", [1.0, 1e-3])
def test_period_maps_and_basins(eng, prec, scale):
    both(eng.run_bif2d, lambda body: ucb.Engine.bif2d_request(
        body, 3, tiny(prec, scale), VALUES, eps_dbscan=0.1, t_max=30.0, **plane(20, prec)))
    x = tiny(prec, scale)[0]
    window = dict(n_pts=20, axis_x_lo=-x, axis_x_hi=x, axis_y_lo=0.01 * x, axis_y_hi=x, opt=options(prec))
    # (an attractor's point is that of the cell that registers it first)
    both(lambda req: (lambda r: r[:3] + r[-1:])(eng.run_basins(req)), lambda body: ucb.Engine.basins_request(
        body, 3, (0.0, 0.0, x), VALUES, period=0.5, steps_per_period=50, max_periods=90, match_count=20, match_tol=1e-6,
        phase_var=-1, max_value=1e6, **window))
    both(eng.run_basins_dbscan, lambda body: ucb.Engine.basins_dbscan_request(
        body, 3, (0.0, 0.0, x), VALUES, h=0.01, t_max=10.0, transient_time=5.0, eps_dbscan=0.5, **window))


def test_settled_lanes_do_not_slow_the_others(eng):
    """FP32 calls some of whose cells settle: with the settled lanes alone on the division a warp paid for
    both passes, 1.28 (map) and 1.18 (diagram) times the verbatim body's time; with the warp together
    1.08 and 1.04, the pass being taken from local memory. The line is drawn between the two. (Kernel
    times, alternating, the better of five.)"""
    wide = dict(transient_time=100.0, t_max=200.0)

    def lle(body):
        return eng.run_lle2d(ucb.Engine.lle2d_request(body, 3, (0.1, 0.1, 0.1), VALUES, NT=0.1, eps=1e-4,
                                                      **plane(256, "f32", opt=options("f32", lle_method=ucb.LLE_SHADOW),
                                                              **wide)))

    def bif(body):
        return eng.run_bif1d(ucb.Engine.bif1d_request(body, 3, (0.1, 0.1, 0.1), VALUES, max_peaks=64,
                                                      **sweep(1024, "f32", **wide)))

    for run in (lle, bif):
        best = {BODY: np.inf, VERBATIM: np.inf}
        for _ in range(5):
            for body in best:
                best[body] = min(best[body], run(body)[-1].kernel_ms)
        assert best[BODY] < 1.13 * best[VERBATIM], (run.__name__, best[BODY], best[VERBATIM])
