"""Adaptive spectra with a cell on amount_of_x lanes (small maps) against a cell a lane (large
maps): the cells two maps share have the same bits, flags and attempts."""
import numpy as np
import pytest

import ucb
from helpers import CHEN, HYPER_ROSSLER, rk4_body

pytestmark = pytest.mark.gpu

SYSTEMS = {  # body, variables, initial conditions, values, swept parameters with windows
    4: (HYPER_ROSSLER, (-10.0, -6.0, 0.0, 10.0), (0, 0.25, 0.05), (1, 0.1, 0.35), (2, 0.01, 0.1)),
    3: (CHEN, (1.0, 1.0, 1.0), (0, 35.0, 3.0, 28.0), (1, 30.0, 40.0), (3, 20.0, 30.0)),
}


def spectrum(eng, nx, n, prec, lo, hi, lo2, hi2, **kw):
    name, ic, values, (p1, _, _), (p2, _, _) = SYSTEMS[nx]
    req = ucb.Engine.ls2d_request(rk4_body(name), nx, ic, values, method=ucb.LS_DP5, n_pts=n, param_index=p1,
                                  param_index_2=p2, param_lo=lo, param_hi=hi, param_lo_2=lo2, param_hi_2=hi2, h=0.01,
                                  NT=1.0, eps=1e-6, opt=ucb.options(precision=prec), **kw)
    v, f, res = eng.run_ls2d(req, cell_steps=True)
    return v, f, res.cell_work


@pytest.mark.parametrize("nx", [4, 3])
@pytest.mark.parametrize("prec,large", [(ucb.PREC_F64, 121), (ucb.PREC_F32, 301)])
@pytest.mark.parametrize("kw", [dict(t_max=3.0, gs_every=10, max_steps=3000),
                                dict(t_max=2.0, transient_time=1.5, gs_every=3, max_steps=400),
                                dict(t_max=4.0, gs_every=1, max_steps=2000, max_value=60.0)])
def test_small_maps_equal_the_large_one(nx, prec, large, kw):
    """Grids of 1, 2, 11, 25 and 61 points an axis take 1 to 10 cells a warp. The probe
    directions are drawn by cell index, so the cells compared are those of the first rows,
    where their axis values agree. Cells end by t_end, the attempt cap, max_value and the
    escape test."""
    _, _, _, (_, lo, hi), (_, lo2, hi2) = SYSTEMS[nx]
    eng = ucb.Engine(0)
    kw = dict(dict(max_value=1e6), **kw)
    v, f, work = spectrum(eng, nx, large, prec, lo, hi, lo2, hi2, **kw)
    v, f, work = v.reshape(nx, large, large), f.reshape(large, large), work.reshape(large, large)
    assert (f == 1).any() or kw["max_steps"] == 400  # (all of Chen at the cap)
    for n in (1, 2, 11, 25, 61):
        # a map of n x n cells whose first row sweeps the large map's first n values
        t = np.float32 if prec == ucb.PREC_F32 else np.float64
        w = t(n - 1) / t(large - 1)
        end = float((t(1) - w) * t(lo) + w * t(hi))
        sv, sf, swork = spectrum(eng, nx, n, prec, lo, end, lo2, hi2 if n > 1 else lo2, **kw)
        big = axis(large, lo, hi, t)[:n]
        small = axis(n, lo, end, t)
        same = np.flatnonzero(big == small)
        assert 0 in same
        sv = sv.reshape(nx, n, n)
        for i in same:
            np.testing.assert_array_equal(sv[:, 0, i], v[:, 0, i])
            assert sf[i] == f[0, i] and swork[i] == work[0, i]
    eng.close()


def axis(n, lo, hi, t):
    """The engine's axis values."""
    lo, hi = t(lo), t(hi)
    if n == 1:
        return np.array([hi])
    return np.array([(t(1) - t(i) / t(n - 1)) * lo + t(i) / t(n - 1) * hi for i in range(n)])
