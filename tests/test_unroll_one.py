"""A caller's unroll of one is taken where a build by itself unrolls its step loop by more (the
stroboscopic basins' table loop by eight, shared forcing phases by four): the program is shorter."""
import numpy as np
import pytest

import ucb
from helpers import DUFFING, rk4_body


def request(call, unroll):
    args = (rk4_body(DUFFING), 3, (0.0, 0.0, 0.0), (0.0,))
    opt = ucb.options(precision=ucb.PREC_F64, unroll=unroll)
    if call == "basins":
        return ucb.Engine.basins_request(*args, n_pts=8, phase_var=2, period=2 * np.pi, opt=opt)
    return ucb.Engine.basins_dbscan_request(*args, n_pts=8, opt=opt)


@pytest.mark.parametrize("call", ["basins", "basins_dbscan"])
def test_program_is_shorter(call, tmp_path, monkeypatch):
    size = {}
    for unroll in (0, 1):
        cache = tmp_path / str(unroll)
        monkeypatch.setenv("UCB_CUBIN_CACHE", str(cache))
        ucb.precompile(request(call, unroll))
        (file,) = cache.iterdir()
        size[unroll] = file.stat().st_size
    assert size[1] < 0.9 * size[0]
