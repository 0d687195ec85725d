"""Shadow maps with a trajectory a lane (few cells) against the pair form (many cells): the
cells of a large map that a small one shares have the same bits."""
import numpy as np
import pytest

import ucb
from helpers import engine_request, lle2d_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,prec", [(ucb.MODE_NATIVE, ucb.PREC_F64), (ucb.MODE_EXACT, ucb.PREC_F64),
                                       (ucb.MODE_EXACT, ucb.PREC_F32)])
@pytest.mark.parametrize("NT,nominal", [(0.1, False), (0.1, True), (0.01, False), (1.57, False)])
@pytest.mark.parametrize("max_value", [1e6, 14.0, 6.0])
def test_listed_cells_equal_the_map(mode, prec, NT, nominal, max_value):
    """The map's own launch takes the pair form; a list of 1, 15, 16, 17 or 100 of its cells
    takes the split form (part-filled warps, neighbouring cells of one warp ending at
    different times, block lengths of one step, a whole unrolled block and over the
    divergence test's interval)."""
    import torch
    c = lle2d_case(n=150, t_max=9.5, transient=3.3, NT=NT, max_value=max_value)
    req = engine_request(ucb, c, precision=prec, mode=mode, nominal_steps=nominal, lle_method=ucb.LLE_SHADOW)
    eng = ucb.Engine(0)
    values, flags, res = eng.run_lle2d(req)
    if max_value == 6.0:
        assert 0 < (flags == -1).sum() < flags.size
    rng = np.random.default_rng(3)
    for n in (1, 15, 16, 17, 100):
        cells = np.sort(rng.choice(values.size, n, replace=False))
        d_cells = torch.from_numpy(cells).cuda()
        v = torch.empty(n, dtype=torch.float64, device="cuda")
        f = torch.empty(n, dtype=torch.int32, device="cuda")
        eng.lle2d_cells(req, d_cells.data_ptr(), n, v.data_ptr(), f.data_ptr(), 0)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(v.cpu().numpy(), values[cells])
        np.testing.assert_array_equal(f.cpu().numpy(), flags[cells])
    eng.close()
