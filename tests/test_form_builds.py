"""The sizes at which other tests compare two forms of a kernel with each other are on both sides of
the line between them: the two sizes are different builds (files of a fresh CUBIN cache)."""
import pytest

import ucb
from helpers import HYPER_ROSSLER, LORENZ, rk4_body

F64, F32 = ucb.PREC_F64, ucb.PREC_F32


def build(cache, request):
    """The cache's file of this request's build."""
    before = {p.name for p in cache.iterdir()} if cache.exists() else set()
    ucb.precompile(request)
    return {p.name for p in cache.iterdir()} - before


def spectrum(method, n, prec, mode=ucb.MODE_NATIVE):
    kw = dict(method=method, t_end=2.0) if method == ucb.LS_DP5 else dict(method=method, NT=0.1)
    return ucb.Engine.ls2d_request(rk4_body(HYPER_ROSSLER), 4, (-10.0, -6.0, 0.0, 10.0), (0, 0.25, 0.05), n_pts=n,
                                   param_index=1, param_index_2=2, param_lo=0.24, param_hi=0.26, param_lo_2=0.045,
                                   param_hi_2=0.055, h=0.01, t_max=2.0, eps=1e-6,
                                   opt=ucb.options(precision=prec, mode=mode), **kw)


def diagram(n, prec, mode, block):
    return ucb.Engine.bif1d_request(rk4_body(LORENZ), 3, (0.1, 0.1, 0.1), (0, 10.0, 28.0, 8 / 3), n_pts=n, param_index=2,
                                    param_lo=20.0, param_hi=200.0, h=0.01, t_max=2.0,
                                    opt=ucb.options(precision=prec, mode=mode, block_threads=block))


FORMS = [("adaptive f64", lambda n: spectrum(ucb.LS_DP5, n, F64), 61, 121),
         ("adaptive f32", lambda n: spectrum(ucb.LS_DP5, n, F32), 61, 301)]
for prec in (F64, F32):
    for mode in (ucb.MODE_NATIVE, ucb.MODE_EXACT):
        FORMS.append((f"fixed {prec} {mode}", lambda n, p=prec, m=mode: spectrum(ucb.LS_FIXED, n, p, m), 33, 400))
        FORMS.append((f"diagram {prec} {mode}", lambda n, p=prec, m=mode: diagram(n, p, m, 0), 9472, 9473))


@pytest.mark.parametrize("name,request_of,few,many", FORMS, ids=[f[0] for f in FORMS])
def test_sizes_on_both_sides(name, request_of, few, many, tmp_path, monkeypatch):
    monkeypatch.setenv("UCB_CUBIN_CACHE", str(tmp_path))
    assert len(build(tmp_path, request_of(few))) == 1
    assert len(build(tmp_path, request_of(few - 1))) == 0  # one build for a form's sizes
    assert len(build(tmp_path, request_of(many))) == 1
