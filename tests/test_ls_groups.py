"""Fixed-step spectra with a cell on several lanes (small maps) against a cell a lane (large
maps): cells that two maps share have the same bits, flags and step counts."""
import numpy as np
import pytest

import ucb
from helpers import HYPER_ROSSLER, LORENZ, rk4_body

pytestmark = pytest.mark.gpu

SYSTEMS = {4: (HYPER_ROSSLER, (-10.0, -6.0, 0.0, 10.0), (0, 0.25, 0.05), 1, 2, 0.24, 0.045, 0.055),
           3: (LORENZ, (0.1, 0.1, 0.1), (0, 10.0, 28.0, 8 / 3), 2, 1, 20.0, 5.0, 15.0)}


@pytest.mark.parametrize("nx", [4, 3])
@pytest.mark.parametrize("prec,mode", [(ucb.PREC_F64, ucb.MODE_NATIVE), (ucb.PREC_F64, ucb.MODE_EXACT),
                                       (ucb.PREC_F32, ucb.MODE_NATIVE), (ucb.PREC_F32, ucb.MODE_EXACT)])
@pytest.mark.parametrize("kw", [dict(NT=0.1, transient_time=2.0), dict(NT=0.01), dict(NT=1.37, transient_time=0.5),
                                dict(NT=0.1, max_value=27.0), dict(NT=1.37, max_value=27.0, nominal=True)])
def test_first_rows_agree(nx, prec, mode, kw):
    """The first axis sweeps one value, so the first n cells of an n x n map are the first n of
    every larger one (the probe directions are drawn by cell index): n = 1, 5, 7 and 33
    (part-filled warps) take groups, 400 a cell a lane. Block lengths of one step, of a whole
    unrolled block and over the divergence test's interval; max_value ends some cells."""
    name, ic, values, p1, p2, lo, lo2, hi2 = SYSTEMS[nx]
    kw = dict(dict(max_value=1e6, transient_time=0.0), **kw)
    opt = ucb.options(precision=prec, mode=mode, nominal_steps=kw.pop("nominal", False))
    eng = ucb.Engine(0)

    def run(n):
        req = ucb.Engine.ls2d_request(rk4_body(name), nx, ic, values, n_pts=n, param_index=p1, param_index_2=p2,
                                      param_lo=lo, param_hi=lo, param_lo_2=lo2, param_hi_2=lo2, h=0.01, t_max=2.8,
                                      eps=1e-6, opt=opt, **kw)
        v, f, res = eng.run_ls2d(req, cell_steps=True)
        return v, f, res.cell_work

    # every cell has the same parameters up to the rounding of (1 - t) v + t v; the probe
    # directions differ from cell to cell
    t = np.float32 if prec == ucb.PREC_F32 else np.float64

    def axis(n, v):
        v = t(v)
        return np.array([v] if n == 1 else [(t(1) - t(i) / t(n - 1)) * v + t(i) / t(n - 1) * v for i in range(n)])

    v, f, work = run(400)
    for n in (1, 5, 7, 33):
        sv, sf, swork = run(n)
        idx = np.arange(n * n)
        a, b = (axis(n, lo)[idx % n], axis(n, lo2)[idx // n]), (axis(400, lo)[idx % 400], axis(400, lo2)[idx // 400])
        same = np.flatnonzero((a[0] == b[0]) & (a[1] == b[1]))
        assert len(same) >= n * n / 3
        np.testing.assert_array_equal(sv[:, same], v[:, same])
        np.testing.assert_array_equal(sf[same], f[same])
        np.testing.assert_array_equal(swork[same], work[same])
    eng.close()
