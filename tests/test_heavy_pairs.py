"""The clustering's search of large square pairs (part boxes, then the cells of the parts about
eps apart) against the reference's literal loop."""
import numpy as np
import pytest

import ucb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [ucb.PREC_F64, ucb.PREC_F32])
@pytest.mark.parametrize("cells", [24, 26, 40, 64])
@pytest.mark.parametrize("gap", [0.98, 1.0 - 1e-6, 1.0, 1.0 + 1e-6, 1.02])
@pytest.mark.parametrize("offset", [0.0, -37.25, 3e7])
def test_facing_arcs(prec, cells, gap, offset):
    """A spot and an arc around it of radius gap x eps (one pair of squares after the other
    holds both): pairs of cells just within, at and just beyond eps in every direction, pair
    products below and above the size the parts are used from, coordinates that resolve the
    parts and (3e7) coordinates that do not."""
    eps, n = 0.5, cells
    m = n * n
    rng = np.random.default_rng(int(cells * 1000 + gap * 100))
    phi = rng.uniform(0, 2 * np.pi, m)
    arc = np.arange(m) % 2 == 1
    r = np.where(arc, gap * eps * (1 + 1e-3 * rng.random(m)), 1e-4 * eps * rng.random(m))
    r[1] = gap * eps  # one cell of the arc exactly on the radius, facing the spot's first
    phi[1] = 0.0
    r[0] = 0.0
    f1, f2 = offset + r * np.cos(phi), offset + r * np.sin(phi)
    cls = rng.choice([-1, 1], m, p=[0.01, 0.99]).astype(np.int32)
    eng = ucb.Engine(0)
    lab, _ = eng.run_basins_recluster("x", 3, n, eps, f1, f2, cls, opt=ucb.options(precision=prec))
    eng.close()
    np.testing.assert_array_equal(lab, O.dbscan_cells(f1, f2, cls, eps, "f64" if prec == ucb.PREC_F64 else "f32"))
