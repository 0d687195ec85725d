"""A run's progress starts at its own beginning: while its inputs still wait for the copy engine, the
work counter in the workspace is that of the call before, and is not reported."""
import ctypes as C
import threading

import pytest

import ucb
from helpers import DUFFING, HYPER_ROSSLER, LORENZ, engine_request, lle2d_case, rk4_body

pytestmark = pytest.mark.gpu


def requests(call):
    """A short run that leaves its counter at the end of a large queue, and a longer one."""
    f64 = ucb.options(precision=ucb.PREC_F64)
    if call == "run_lle2d":
        return [engine_request(ucb, lle2d_case(n=600, t_max=t, transient=1.0), precision=ucb.PREC_F64)
                for t in (2.0, 60.0)]
    lorenz = (rk4_body(LORENZ), 3, (0.1, 0.1, 0.1), (0, 10.0, 28.0, 8 / 3))
    plane = dict(param_index=2, param_index_2=1, param_lo=20.0, param_hi=200.0, param_lo_2=5.0, param_hi_2=15.0, h=0.01,
                 opt=f64)
    if call == "run_bif2d":
        return [ucb.Engine.bif2d_request(*lorenz, n_pts=600, t_max=t, eps_dbscan=0.1, **plane) for t in (1.0, 30.0)]
    if call == "run_ls2d":
        return [ucb.Engine.ls2d_request(rk4_body(HYPER_ROSSLER), 4, (-10.0, -6.0, 0.0, 10.0), (0, 0.25, 0.05),
                                        method=ucb.LS_FIXED, n_pts=500, param_index=1, param_index_2=2, param_lo=0.24,
                                        param_hi=0.26, param_lo_2=0.045, param_hi_2=0.055, h=0.01, NT=0.1, eps=1e-6,
                                        t_max=t, opt=f64) for t in (1.0, 15.0)]
    duffing = (rk4_body(DUFFING), 3, (0.0, 0.0, 0.0), (0.0,))
    window = dict(n_pts=600, axis_x_lo=-2.5, axis_x_hi=2.5, axis_y_lo=-2.5, axis_y_hi=2.5, opt=f64)
    if call == "run_basins":
        return [ucb.Engine.basins_request(*duffing, period=6.28, steps_per_period=100, max_periods=p, phase_var=2,
                                          **window) for p in (4, 130)]
    return [ucb.Engine.basins_dbscan_request(*duffing, h=0.03, t_max=t, transient_time=1.0, eps_dbscan=0.5, **window)
            for t in (1.0, 60.0)]


@pytest.mark.parametrize("call", ["run_lle2d", "run_bif2d", "run_ls2d", "run_basins", "run_basins_dbscan"])
def test_first_progress_is_not_the_last_calls(call):
    import torch
    eng = ucb.Engine(0)
    short, long = requests(call)
    run = getattr(eng, call)
    run(long)
    # uploads of this stream queue before the run's own
    host = torch.empty(1 << 27, dtype=torch.float32, pin_memory=True)
    dev = torch.empty(1 << 27, dtype=torch.float32, device="cuda")
    for _ in range(3):
        run(short)
        prog, phase = C.c_float(-1.0), C.c_int32(0)
        long.progress = C.pointer(prog)
        if hasattr(long, "progress_phase"):
            long.progress_phase = C.pointer(phase)
        seen, done = [], threading.Event()

        def watch():
            while not done.is_set():
                value = prog.value
                if phase.value < 2:  # (of the map itself, not the clustering after it)
                    seen.append(value)

        torch.cuda.synchronize()
        for _ in range(4):
            dev.copy_(host, non_blocking=True)
        thread = threading.Thread(target=watch)
        thread.start()
        run(long)
        done.set()
        thread.join()
        seen = [p for p in seen if 0.0 <= p < 1.0]
        assert any(p > 0 for p in seen)
        assert all(b >= a for a, b in zip(seen, seen[1:])), [a for a, b in zip(seen, seen[1:]) if b < a]
    eng.close()
