"""Diagrams with two warps for 32 points (the default for few points) against one warp doing
both (blocks of 128 threads): the same counts, peaks, intervals and steps."""
import numpy as np
import pytest

import ucb
from helpers import LORENZ, rk4_body

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [ucb.PREC_F64, ucb.PREC_F32])
@pytest.mark.parametrize("mode", [ucb.MODE_NATIVE, ucb.MODE_EXACT])
@pytest.mark.parametrize("kw", [
    dict(n_pts=1), dict(n_pts=31), dict(n_pts=33), dict(n_pts=100, max_peaks=3), dict(n_pts=40, writable_var=-1),
    dict(n_pts=40, pre_scaller=3, writable_var=2), dict(n_pts=40, max_value=45.0), dict(n_pts=40, max_value=80.0),
    dict(n_pts=70, sweep_over_h=True, param_lo=0.004, param_hi=0.02),
    dict(n_pts=70, sweep_over_var=True, var_sweep_index=0, param_lo=-9.0, param_hi=9.0)]
    + [dict(n_pts=34, t_max=t) for t in (0.01, 0.04, 0.05, 0.24, 0.25, 0.26, 0.5, 0.99, 1.0, 1.01, 1.25)])
def test_two_warps_equal_one(prec, mode, kw):
    """Part-filled warps, points that diverge before and during the record, points of unequal
    length (h sweep), horizons around the chunk and the divergence test's interval."""
    eng = ucb.Engine(0)
    out = []
    for block in (0, 64, 128):
        base = dict(param_index=2, param_lo=20.0, param_hi=200.0, h=0.01, transient_time=1.7, t_max=12.0, max_peaks=40,
                    max_value=1e6)
        req = ucb.Engine.bif1d_request(rk4_body(LORENZ), 3, (0.1, 0.1, 0.1), (0, 10.0, 28.0, 8 / 3),
                                       opt=ucb.options(precision=prec, mode=mode, block_threads=block),
                                       **dict(base, **kw))
        out.append(eng.run_bif1d(req))
    eng.close()
    for other in out[1:]:
        for a, b in zip(out[0][:3], other[:3]):
            np.testing.assert_array_equal(a, b)
        assert out[0][3].steps == other[3].steps
