"""Measured calls of the engine: one dict per case, run through the public Python binding.

The cases are the calls a session makes: one-dimensional curves and two-dimensional maps of
the largest exponent, bifurcation diagrams and period maps, Lyapunov spectra, basins of
attraction by both methods, the clustering alone, and the surrogate network's two
directions. Systems, windows and horizons are those of bench.py's configurations; grids
run from a curve of a few hundred points to the 1024 x 1024 map. The seed moves every window
and initial condition a little, so that no two seeds integrate the same cells.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "u-cuda_b200"))

import ucb  # noqa: E402

# text, alphabet, state size, initial conditions, parameter vector a[] (a[0] is reserved),
# the two swept parameters with their windows, FLOPs of one right-hand side and of one J v
# product (fused multiply-add = 2).
SYSTEMS = {
    "rossler": dict(text=r"\dot{x} = -y-z \\ \dot{y} = x + a y \\ \dot{z} = b + z(x-c)", alphabet="x,y,z,a,b,c", nx=3,
                    ic=(1.0, 1.0, 1.0), values=(0.0, 0.2, 0.2, 5.7), sweep=((2, 0.05, 2.0), (3, 2.0, 20.0)), h=0.01,
                    rhs=7, jvp=8),
    "lorenz": dict(text=r"\dot{x} = s (y-x) \\ \dot{y} = x (r-z) - y \\ \dot{z} = x y - b z", alphabet="x,y,z,s,r,b",
                   nx=3, ic=(0.1, 0.1, 0.1), values=(0.0, 10.0, 28.0, 8.0 / 3.0),
                   sweep=((2, 20.0, 200.0), (1, 5.0, 15.0)), h=0.01, rhs=8, jvp=11),
    "chen": dict(text=r"\dot{x} = a(y-x) \\ \dot{y} = (c-a)x - x z + c y \\ \dot{z} = x y - b z",
                 alphabet="x,y,z,a,b,c", nx=3, ic=(1.0, 1.0, 1.0), values=(0.0, 35.0, 3.0, 28.0),
                 sweep=((1, 30.0, 40.0), (3, 20.0, 30.0)), h=0.002, rhs=11, jvp=14),
    "hyper_rossler": dict(text=r"\dot{x} = -y-z \\ \dot{y} = x + p y + w \\ \dot{z} = 3 + x z \\ \dot{w} = -0.5 z + q w",
                          alphabet="x,y,z,w,p,q", nx=4, ic=(-10.0, -6.0, 0.0, 10.0), values=(0.0, 0.25, 0.05),
                          sweep=((1, 0.24, 0.26), (2, 0.045, 0.055)), h=0.01, rhs=9, jvp=10),
    "duffing": dict(text=r"\dot{x} = v \\ \dot{v} = -0.15 v + x - x^{3} + 0.3\cos(s) \\ \dot{s} = 1", alphabet="x,v,s",
                    nx=3, ic=(0.0, 0.0, 0.0), values=(0.0,), sweep=(), h=2 * math.pi / 200, rhs=9, jvp=10),
}
FOURIER = 64  # frequencies of the surrogate network's input features


def listed():
    return [
        # the curve a user drags a slider over: few trajectories, so one trajectory's latency
        dict(name="lle1d_f64_exact_200", call="lle1d", system="rossler", n=200, precision="f64", mode="exact",
             transient=50.0, t_max=200.0),
        # the headline map: largest exponent over 1024 x 1024 cells in the FP32 form, kept in HBM
        dict(name="lle2d_f32_1024", call="lle2d", system="rossler", n=1024, precision="f32", mode="native",
             sweep="params", device=True, transient=100.0, t_max=1000.0),
        # the plain FP64 map at a figure's size, to host memory
        dict(name="lle2d_f64_300", call="lle2d", system="chen", n=300, precision="f64", mode="native", sweep="params",
             device=False, transient=20.0, t_max=100.0),
        # the bifurcation diagram of the reference's front page: 1024 values, every maximum
        dict(name="bif1d_f64_1024", call="bif1d", system="lorenz", n=1024, precision="f64", mode="native",
             transient=50.0, t_max=200.0, max_peaks=64),
        # the period map: peaks of every cell clustered
        dict(name="bif2d_f64_256", call="bif2d", system="lorenz", n=256, precision="f64", mode="native",
             transient=50.0, t_max=200.0, eps=0.1),
        # the whole spectrum by the reference's fixed-step method
        dict(name="ls2d_f64_256", call="ls2d", system="hyper_rossler", n=256, precision="f64", mode="native",
             transient=10.0, t_max=100.0),
        # the whole spectrum with adaptive steps over the wide window, where cells stop early or late
        dict(name="ls2d_dp5_f64_96", call="ls2d_dp5", system="hyper_rossler", n=96, precision="f64", t_end=50.0,
             max_steps=20000),
        # basins by stroboscopic labels
        dict(name="basins_f64_512", call="basins", system="duffing", n=512, precision="f64", max_periods=2000),
        # basins by the reference's method: features of every cell, then the clustering
        dict(name="basins_dbscan_f32_256", call="basins_dbscan", system="duffing", n=256, precision="f32",
             transient=10000.0, t_max=1000.0, eps=0.5),
        # the clustering again with another eps, over the features of a finished map
        dict(name="recluster_f64_1024", call="recluster", n=1024, precision="f64", eps=0.25, attractors=4),
        # the surrogate network over every cell of a 1024 x 1024 map
        dict(name="mlp_predict_1048576", call="predict", rows=1 << 20, layers=4, hidden=256),
        # its training on the samples of a 256 x 256 partition
        dict(name="mlp_fit_8192x100", call="fit", rows=65536, batch=8192, steps=100, layers=4, hidden=256),
    ]


def _between(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _real(rng, lo, hi):
    return round(math.exp(rng.uniform(math.log(lo), math.log(hi))), 4)


def draw(rng):
    call = rng.choice(["lle1d", "lle2d", "bif1d", "bif2d", "ls2d", "ls2d_dp5", "basins", "basins_dbscan", "recluster",
                       "predict", "fit"])
    prec = rng.choice(["f64", "f32"])
    mode = rng.choice(["native", "native", "exact"])
    system = rng.choice(["rossler", "lorenz", "chen"])
    span = 0.2 if system == "chen" else 1.0  # its step is a fifth of the others'
    if call == "lle1d":
        return dict(call=call, system=system, n=_between(rng, 64, 2048), precision=prec, mode=mode,
                    transient=_real(rng, 20, 100) * span, t_max=_real(rng, 50, 400) * span)
    if call == "lle2d":
        return dict(call=call, system=system, n=_between(rng, 48, 600), precision=prec, mode=mode,
                    sweep=rng.choice(["params", "params", "states"]), device=rng.choice([True, False]),
                    transient=_real(rng, 20, 100) * span, t_max=_real(rng, 50, 400) * span)
    if call == "bif1d":
        return dict(call=call, system=system, n=_between(rng, 100, 4096), precision=prec, mode=mode,
                    transient=_real(rng, 20, 100) * span, t_max=_real(rng, 50, 300) * span,
                    max_peaks=rng.choice([32, 64, 200]))
    if call == "bif2d":
        return dict(call=call, system=system, n=_between(rng, 32, 300), precision=prec, mode=mode,
                    transient=_real(rng, 20, 100) * span, t_max=_real(rng, 50, 300) * span, eps=_real(rng, 0.02, 0.5))
    if call == "ls2d":
        return dict(call=call, system=rng.choice(["hyper_rossler", "lorenz", "rossler"]), n=_between(rng, 32, 300),
                    precision=prec, mode=mode, transient=_real(rng, 5, 30), t_max=_real(rng, 30, 150))
    if call == "ls2d_dp5":
        return dict(call=call, system="hyper_rossler", n=_between(rng, 16, 128), precision=prec,
                    t_end=_real(rng, 10, 80), max_steps=20000)
    if call == "basins":
        return dict(call=call, system="duffing", n=_between(rng, 48, 640), precision=prec,
                    max_periods=rng.choice([500, 1000, 2000]))
    if call == "basins_dbscan":
        return dict(call=call, system="duffing", n=_between(rng, 32, 320), precision=prec,
                    transient=_real(rng, 300, 10000), t_max=_real(rng, 200, 1000), eps=_real(rng, 0.1, 1.0))
    if call == "recluster":
        return dict(call=call, n=_between(rng, 64, 1100), precision=prec, eps=_real(rng, 0.1, 0.6),
                    attractors=rng.randint(1, 12))
    if call == "predict":
        return dict(call=call, rows=_between(rng, 500, 1 << 20), layers=rng.randint(2, 5), hidden=rng.choice([128, 256]))
    return dict(call=call, rows=_between(rng, 1024, 65536), batch=128 * _between(rng, 8, 64), steps=_between(rng, 20, 120),
                layers=rng.randint(2, 5), hidden=rng.choice([128, 256]))


_BODIES = {}
_ENGINE = []


def _engine():
    """The engine a program holds for its whole life (one per device)."""
    if not _ENGINE:
        _ENGINE.append(ucb.Engine(0))
    return _ENGINE[0]


def _body(system):
    if system not in _BODIES:
        s = SYSTEMS[system]
        _BODIES[system] = ucb.codegen(s["text"], s["alphabet"], "RK4")[0]
    return _BODIES[system]


def _options(case):
    return ucb.options(precision=ucb.PREC_F32 if case["precision"] == "f32" else ucb.PREC_F64,
                       mode=ucb.MODE_EXACT if case.get("mode") == "exact" else ucb.MODE_NATIVE)


def _window(rng, lo, hi):
    """The window moved by up to 1 % of its width at both ends."""
    w = hi - lo
    return lo + 0.01 * w * rng.random(), hi - 0.01 * w * rng.random()


def _network(case, seed):
    return ucb.Mlp(_engine(), fourier=FOURIER, hidden=case["hidden"], layers=case["layers"], seed=seed % (1 << 31),
                   batch=case.get("batch", 8192), train_steps=case.get("steps", 0))


def _inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    u = torch.rand(case["rows"], 2, generator=g, device="cuda")
    # a smooth exponent surface with the per-cell noise of the random probe direction
    y = 0.4 * torch.sin(5.0 * u[:, 0]) * torch.cos(3.0 * u[:, 1]) + 0.2 * u[:, 0] - 0.1
    return u, y + 0.01 * torch.randn(case["rows"], generator=g, device="cuda")


def _features(case, rng):
    """Features and classes of a finished map as basins of several attractors give them:
    per attractor a dense spot of (mean peak, mean interval), from a periodic orbit's few
    thousandths to a chaotic set's few tenths wide; some cells rest at a fixed point or escape."""
    n, k = case["n"] ** 2, case["attractors"]
    owner = rng.integers(0, k, n)
    centre = rng.uniform(-4.0, 4.0, (k, 2))
    width = np.exp(rng.uniform(np.log(0.003), np.log(0.4), (k, 2)))
    f = centre[owner] + width[owner] * rng.standard_normal((n, 2))
    cls = np.ones(n, dtype=np.int32)
    fate = rng.random(n)
    fixed, unbound = fate < 0.05, fate > 0.98
    f[fixed] = np.stack([np.where(owner[fixed] % 2 == 0, 1.0, -1.0), np.full(fixed.sum(), -1.0)], axis=1)
    f[unbound] = 999.0
    cls[fixed], cls[unbound] = -1, 0
    return np.ascontiguousarray(f[:, 0]), np.ascontiguousarray(f[:, 1]), cls


def prepare(case, seed):
    rng = np.random.default_rng(int(seed))
    call = case["call"]
    state = dict(call=call, engine=_engine())
    if call in ("predict", "fit"):
        net = _network(case, seed)
        u, y = _inputs(case, seed)
        state.update(net=net, u=u, y=y, start=net.get_params(), mean=torch.empty(case["rows"], device="cuda"),
                     std=torch.empty(case["rows"], device="cuda"))
        return state
    if call == "recluster":
        f1, f2, cls = _features(case, rng)
        state.update(args=("X[0] = X[0];", 3, case["n"], case["eps"], f1, f2, cls), opt=_options(case))
        return state
    s = SYSTEMS[case["system"]]
    ic = tuple(v + 1e-3 * rng.random() for v in s["ic"])
    opt = _options(case)
    base = (_body(case["system"]), s["nx"], ic, s["values"])
    if call == "basins":
        lo, hi = _window(rng, -2.5, 2.5)
        lo2, hi2 = _window(rng, -2.5, 2.5)
        state["req"] = ucb.Engine.basins_request(
            *base[:2], s["ic"], s["values"], n_pts=case["n"], axis_x_var=0, axis_y_var=1, axis_x_lo=lo, axis_x_hi=hi,
            axis_y_lo=lo2, axis_y_hi=hi2, period=2 * math.pi, steps_per_period=200, max_periods=case["max_periods"],
            match_count=20, match_tol=1e-6, phase_var=2, max_value=1e6, opt=opt)
        return state
    if call == "basins_dbscan":
        lo, hi = _window(rng, -2.5, 2.5)
        lo2, hi2 = _window(rng, -2.5, 2.5)
        state["req"] = ucb.Engine.basins_dbscan_request(
            *base[:2], s["ic"], s["values"], n_pts=case["n"], axis_x_lo=lo, axis_x_hi=hi, axis_y_lo=lo2, axis_y_hi=hi2,
            h=s["h"], t_max=case["t_max"], transient_time=case["transient"], eps_dbscan=case["eps"], opt=opt)
        return state
    (p1, lo, hi), (p2, lo2, hi2) = s["sweep"]
    if call == "ls2d_dp5":
        lo, hi, lo2, hi2 = 0.1, 0.35, 0.01, 0.1  # the wide window: most cells leave, at very different times
    lo, hi = _window(rng, lo, hi)
    lo2, hi2 = _window(rng, lo2, hi2)
    one = dict(n_pts=case["n"], param_index=p1, param_lo=lo, param_hi=hi, h=s["h"], max_value=1e6, opt=opt)
    two = dict(one, param_index_2=p2, param_lo_2=lo2, param_hi_2=hi2)
    times = dict(transient_time=case.get("transient", 0.0), t_max=case.get("t_max", 0.0))
    if call == "lle1d":
        state["req"] = ucb.Engine.lle1d_request(*base, NT=10 * s["h"], eps=1e-4, **times, **one)
    elif call == "lle2d":
        if case["sweep"] == "states":  # the map over two initial conditions
            two.update(sweep_over_var=True, sweep_over_var_2=True, var_sweep_index=0, var_sweep_index_2=1,
                       param_index=0, param_index_2=0, param_lo=lo * 0.01, param_hi=1.0 + rng.random(),
                       param_lo_2=-1.0, param_hi_2=1.0 + rng.random())
        state["req"] = ucb.Engine.lle2d_request(*base, NT=10 * s["h"], eps=1e-4, **times, **two)
        if case["device"]:
            state["values"] = torch.empty(case["n"] ** 2, dtype=torch.float64, device="cuda")
            state["flags"] = torch.empty(case["n"] ** 2, dtype=torch.int32, device="cuda")
    elif call == "bif1d":
        state["req"] = ucb.Engine.bif1d_request(*base, max_peaks=case["max_peaks"], **times, **one)
    elif call == "bif2d":
        state["req"] = ucb.Engine.bif2d_request(*base, eps_dbscan=case["eps"], **times, **two)
    elif call == "ls2d":
        state["req"] = ucb.Engine.ls2d_request(*base, method=ucb.LS_FIXED, NT=10 * s["h"], eps=1e-6, **times, **two)
    else:
        times = dict(transient_time=0.0, t_max=case["t_end"])
        state["req"] = ucb.Engine.ls2d_request(
            *base, method=ucb.LS_DP5, gs_every=10, rtol=1e-8 if case["precision"] == "f64" else 1e-5,
            t_end=case["t_end"], max_steps=case["max_steps"], NT=1.0, eps=1e-6, **times, **two)
    return state


def run(state):
    eng, call = state["engine"], state["call"]
    if call == "lle1d":
        return eng.run_lle1d(state["req"])[:2]
    if call == "lle2d":
        if "values" not in state:
            return eng.run_lle2d(state["req"])[:2]
        eng.lle2d_device(state["req"], state["values"].data_ptr(), state["flags"].data_ptr(),
                         torch.cuda.current_stream().cuda_stream)
        return state["values"], state["flags"]
    if call == "bif1d":
        return eng.run_bif1d(state["req"])[:3]
    if call == "bif2d":
        return eng.run_bif2d(state["req"])[:2]
    if call in ("ls2d", "ls2d_dp5"):
        return eng.run_ls2d(state["req"])[:2]
    if call == "basins":
        labels, periods, iterations, attractors, _ = eng.run_basins(state["req"])
        return labels, periods, iterations, np.array(attractors, dtype=np.float64).reshape(-1, 3)
    if call == "basins_dbscan":
        return eng.run_basins_dbscan(state["req"])[:4]
    if call == "recluster":
        return eng.run_basins_recluster(*state["args"], opt=state["opt"])[0]
    net, u = state["net"], state["u"]
    if call == "predict":
        net.predict(u.data_ptr(), u.shape[0], state["mean"].data_ptr(), state["std"].data_ptr(),
                    torch.cuda.current_stream().cuda_stream)
        return state["mean"], state["std"]
    net.set_params(state["start"])
    loss = net.fit(u.data_ptr(), state["y"].data_ptr(), u.shape[0], torch.cuda.current_stream().cuda_stream)
    return loss, net.get_params()


def _network_flops(case):
    """Multiply-adds of one row through the network, times two."""
    h = case["hidden"]
    return 2 * (2 * FOURIER * h + (case["layers"] - 1) * h * h + 2 * h)


def work(case):
    call = case["call"]
    if call == "predict":
        return {"bytes": 16 * case["rows"], "flops": case["rows"] * _network_flops(case)}
    if call == "fit":
        # forward, gradients of the activations, gradients of the weights
        return {"bytes": 12 * case["rows"] + 4 * _network_flops(case), "flops": 3 * case["batch"] * case["steps"] *
                _network_flops(case)}
    cells = case["n"] if call in ("lle1d", "bif1d") else case["n"] ** 2
    if call == "recluster":
        return {"bytes": 24 * cells, "flops": 5 * cells}
    s = SYSTEMS[case["system"]]
    nx, h = s["nx"], s["h"]
    step = 4 * s["rhs"] + 12 * nx  # one RK4 step of one trajectory
    if call in ("lle1d", "lle2d"):
        # x alone, then x with its shadow or tangent vector; a loop call ends with an extra step
        steps = case["transient"] / h + 2 * 1.1 * case["t_max"] / h
        return {"bytes": 12 * cells, "flops": cells * steps * step}
    if call in ("bif1d", "bif2d"):
        steps = (case["transient"] + case["t_max"]) / h
        return {"bytes": cells * (4 + 16 * case["max_peaks"] if call == "bif1d" else 12), "flops": cells * steps * step}
    if call == "ls2d":
        steps = case["transient"] / h + (nx + 1) * 1.1 * case["t_max"] / h
        return {"bytes": cells * (8 * nx + 4), "flops": cells * steps * step}
    if call == "ls2d_dp5":
        # six stages of x and of nx tangent vectors an attempt; most cells of the window are
        # stiff and take far more attempts than the t_end / h counted here
        attempt = 6 * s["rhs"] + 56 * nx + nx * (6 * s["jvp"] + 40 * nx)
        return {"bytes": cells * (8 * nx + 4), "flops": cells * case["t_end"] / h * attempt}
    if call == "basins":
        # about two thirds of these initial conditions run to the cap
        return {"bytes": 12 * cells, "flops": cells * 0.65 * case["max_periods"] * 200 * step}
    return {"bytes": 24 * cells, "flops": cells * (case["transient"] + case["t_max"]) / h * step}


def exact(case, seed):
    """The network's prediction in 64 bits. A trajectory's exponents, peaks and labels have no
    value that another order of rounding reaches (the systems are chaotic), and a clustering's
    labels are whole numbers."""
    if case["call"] != "predict":
        return None
    net = _network(case, seed)
    u = _inputs(case, seed)[0].double()
    p = torch.from_numpy(net.get_params()).cuda().double()
    freq = torch.from_numpy(net.fourier()).cuda().double()
    net.close()
    mean = torch.empty(u.shape[0], dtype=torch.float64, device="cuda")
    std = torch.empty_like(mean)
    for i in range(0, u.shape[0], 1 << 17):
        z = 2 * math.pi * (u[i:i + (1 << 17)] @ freq.T)
        x = torch.cat([torch.sin(z), torch.cos(z)], dim=1)
        at, width = 0, x.shape[1]
        for layer in range(case["layers"] + 1):
            out = 2 if layer == case["layers"] else case["hidden"]
            w, b = p[at:at + out * width].reshape(out, width), p[at + out * width:at + out * width + out]
            at, width = at + out * width + out, out
            x = x @ w.T + b
            if layer < case["layers"]:
                x = torch.nn.functional.gelu(x, approximate="tanh")
        mean[i:i + (1 << 17)] = x[:, 0]
        std[i:i + (1 << 17)] = torch.exp(0.5 * x[:, 1])
    return mean, std
