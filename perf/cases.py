"""The work a user of this framework has it do, as cases to be timed: parameter
maps through the adaptive sweeps (one model, and mixed batches), the
reference-exact fixed-step sweep behind the drop-in launcher, trajectories,
and the surrogate's training and prediction.

Grids, initial states, tolerances and renormalisation intervals are those of
this repository's benchmark and tests; horizons are shortened (a tenth, mostly)
so that a pass stays below a second.  Inputs are made from the seed with numpy
alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import chaos_oneapi_b200 as cl
from chaos_oneapi_b200.surrogate import MLPEnsemble

# model -> default parameters, the two swept parameters (index, start, end),
# initial state, and attempted steps per unit of time (mean over the map, from
# the kernels' own per-point counters) of Dopri5 rtol 1e-6 and DVERK rtol 1e-10
MODELS = {
    # sigma x rho, the benchmark's Lorenz map
    "lorenz": dict(base=[10.0, 28.0, 8.0 / 3.0], s1=(0, 5.0, 20.0), s2=(1, 0.0, 200.0),
                   x0=[1.0, 1.0, 1.0], rate=(92.0, 320.0), flops=(9, 12)),
    # a x c, the part of the benchmark's Rossler map where orbits stay bounded
    "rossler": dict(base=[0.2, 0.2, 5.7], s1=(0, 0.05, 0.3), s2=(2, 2.0, 12.0),
                    x0=[1.0, 1.0, 0.0], rate=(24.0, 75.0), flops=(7, 8)),
    # alpha x beta, the part of the batch's Chua map where orbits stay bounded
    "chua": dict(base=[9.0, 14.3, -8.0 / 7.0, -5.0 / 7.0], s1=(0, 8.0, 9.1), s2=(1, 12.5, 18.0),
                 x0=[0.1, 0.0, 0.0], rate=(27.0, 100.0), flops=(14, 9)),
    # alpha x lambda, the reference's own model and sweep
    "shimizu": dict(base=[0.0, 0.0], s1=(0, 0.2, 2.0), s2=(1, 0.05, 1.2),
                    x0=[0.1, 0.05, 0.02], rate=(6.0, 20.0), flops=(7, 9)),
    # c x d, a part of the batch's hyperchaotic Rossler map where orbits stay bounded
    "hyper_rossler": dict(base=[0.5, 0.05], s1=(0, 0.41, 0.47), s2=(1, 0.0475, 0.052),
                          x0=[-10.0, -6.0, 0.0, 10.0], rate=(268.0, 900.0), flops=(10, 11)),
    "lorenz96": dict(base=[8.0, 1.0], s1=(0, 4.0, 16.0), s2=(1, 0.5, 1.5), x0=None,
                     rate=(38.0, 100.0), flops=(200, 320)),
}
DOMAIN = (5.0, 20.0, 0.0, 200.0)  # the surrogate's parameter plane: Lorenz sigma x rho


def listed():
    return [
        # the smallest call: a 16 x 16 map of host arrays, short horizon, where
        # copies, launches and one step's latency are the time
        dict(name="host map 16x16", kind="host", model="lorenz", n1=16, n2=16, precision="fp32",
             integrator="dopri5", rtol=1e-6, t_tr=1.0, t_avg=10.0, dt=1.0),
        # the headline: the 1024^2 Lorenz map in the precision form
        dict(name="lorenz 1024 fp32", kind="map", model="lorenz", n1=1024, n2=1024,
             precision="fp32", integrator="dopri5", rtol=1e-6, t_tr=10.0, t_avg=100.0, dt=1.0,
             schedule="auto", block=0, variant=0),
        # the precision form's other map, ragged
        dict(name="rossler 333x257 fp32", kind="map", model="rossler", n1=333, n2=257,
             precision="fp32", integrator="dopri5", rtol=1e-6, t_tr=50.0, t_avg=500.0, dt=2.0,
             schedule="auto", block=0, variant=0),
        # the plain method of the surrogate and of every accuracy check
        dict(name="lorenz 256 fp64", kind="map", model="lorenz", n1=256, n2=256,
             precision="fp64", integrator="dverk65", rtol=1e-10, t_tr=10.0, t_avg=100.0, dt=1.0,
             schedule="auto", block=0, variant=0),
        # a small map in the launch shape the autotuner keeps for it
        dict(name="lorenz 64 fp64 split", kind="map", model="lorenz", n1=64, n2=64,
             precision="fp64", integrator="dverk65", rtol=1e-10, t_tr=30.0, t_avg=300.0, dt=1.0,
             schedule="split_persistent", block=64, variant=1),
        # 40 exponents of the 40-dimensional model
        dict(name="lorenz96 64", kind="map", model="lorenz96", n1=64, n2=64, precision="fp32",
             integrator="dopri5", rtol=1e-6, t_tr=5.0, t_avg=50.0, dt=0.5, schedule="auto",
             block=0, variant=0),
        # three models with averaging times of their own in one replayed graph
        dict(name="batch 3x128", kind="batch", n=128, t_tr=20.0, t_lo=20.0, t_hi=80.0),
        # the reference's default run: its model, FD method, fixed step
        dict(name="compat fd 96x80", kind="compat", model="shimizu", method="fd", n1=96, n2=80,
             h=0.01, t_skip=10.0, t_clp=5.0, t_calc=25.0, t_norm=0.5),
        # the same launcher's QR method, which renormalises every step
        dict(name="compat qr 45x33", kind="compat", model="lorenz", method="qr", n1=45, n2=33,
             h=0.01, t_skip=2.0, t_clp=0.0, t_calc=6.0, t_norm=0.5),
        # trajectories for plots: every accepted step of 8192 orbits
        dict(name="trajectory 8192x500", kind="trajectory", model="lorenz", P=8192, nsteps=500,
             precision="fp64", integrator="dopri5", rtol=1e-8),
        # the surrogate: fitting the coarse sweep, and filling a fine map
        dict(name="surrogate train", kind="train", E=4, W=128, rows=16384, batch=1024, steps=60),
        dict(name="surrogate predict 1M", kind="predict", E=4, W=128, rows=1 << 20),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "map32", "map32", "map64", "split", "lorenz96", "batch", "compat",
                       "compat", "trajectory", "train", "predict"])
    if kind == "host":
        return dict(kind="host", model="lorenz", n1=rng.randint(8, 40), n2=rng.randint(8, 40),
                    precision=rng.choice(["fp32", "fp64"]), integrator="dopri5", rtol=1e-6,
                    t_tr=1.0, t_avg=10.0, dt=1.0)
    if kind == "map32":
        model = rng.choice(["lorenz", "rossler"])
        long = 5.0 if model == "rossler" else 1.0
        return dict(kind="map", model=model, n1=_log_int(rng, 100, 800), n2=_log_int(rng, 100, 800),
                    precision="fp32", integrator=rng.choice(["dopri5", "dopri5", "dverk65"]),
                    rtol=1e-6, t_tr=10.0 * long, t_avg=100.0 * long, dt=1.0 if long == 1 else 2.0,
                    schedule="auto", block=0, variant=rng.choice([0, 0, 1]))
    if kind == "map64":
        return dict(kind="map", model=rng.choice(["lorenz", "rossler"]), n1=_log_int(rng, 100, 256),
                    n2=_log_int(rng, 100, 256), precision="fp64",
                    integrator=rng.choice(["dverk65", "dverk65", "dopri5"]),
                    rtol=rng.choice([1e-10, 1e-8]), t_tr=10.0, t_avg=rng.choice([60.0, 100.0]),
                    dt=1.0, schedule="auto", block=0, variant=0)
    if kind == "split":
        precision = rng.choice(["fp64", "fp64", "fp32"])
        return dict(kind="map", model="lorenz", n1=rng.randint(40, 90), n2=rng.randint(40, 90),
                    precision=precision, integrator="dverk65" if precision == "fp64" else "dopri5",
                    rtol=1e-10 if precision == "fp64" else 1e-6, t_tr=20.0, t_avg=200.0, dt=1.0,
                    schedule="split_persistent", block=rng.choice([0, 64, 128]),
                    variant=rng.choice([0, 1]))
    if kind == "lorenz96":
        return dict(kind="map", model="lorenz96", n1=rng.randint(20, 64), n2=rng.randint(20, 64),
                    precision="fp32", integrator="dopri5", rtol=1e-6, t_tr=5.0,
                    t_avg=rng.choice([20.0, 35.0]), dt=0.5, schedule="auto", block=0, variant=0)
    if kind == "batch":
        return dict(kind="batch", n=rng.randint(50, 128), t_tr=rng.choice([10.0, 20.0]), t_lo=20.0,
                    t_hi=rng.choice([50.0, 65.0, 80.0]))
    if kind == "compat":
        method = rng.choice(["fd", "var", "qr"])
        model = rng.choice(["shimizu", "lorenz"])
        # short of the time in which rounding grows to the size of the orbit
        t_calc = rng.choice([10.0, 15.0, 20.0]) if model == "shimizu" else rng.choice([3.0, 5.0])
        return dict(kind="compat", model=model, method=method, n1=_log_int(rng, 8, 128),
                    n2=_log_int(rng, 8, 128), h=0.01, t_skip=2.0,
                    t_clp=0.0 if method == "qr" else 1.0,
                    t_calc=t_calc, t_norm=rng.choice([0.1, 0.5]))
    if kind == "trajectory":
        return dict(kind="trajectory", model=rng.choice(["lorenz", "rossler"]),
                    P=_log_int(rng, 64, 16384), nsteps=rng.randint(50, 500),
                    precision=rng.choice(["fp64", "fp64", "fp32"]),
                    integrator=rng.choice(["dopri5", "dopri5", "dverk65"]),
                    rtol=1e-6)
    if kind == "train":
        return dict(kind="train", E=rng.choice([2, 4, 5]), W=rng.choice([128, 128, 64]),
                    rows=_log_int(rng, 3000, 40000), batch=rng.choice([1024, 512, 1000]),
                    steps=rng.randint(20, 80))
    return dict(kind="predict", E=rng.choice([2, 4, 5]), W=rng.choice([128, 128, 64]),
                rows=_log_int(rng, 5000, 1 << 20))


# ------------------------------------------------------------------ inputs
def _grid(m, n1, n2):
    """Parameters of the n1 x n2 map, first swept parameter outermost."""
    p = np.tile(np.asarray(m["base"]), (n1 * n2, 1))
    a = np.linspace(m["s1"][1], m["s1"][2], n1)
    b = np.linspace(m["s2"][1], m["s2"][2], n2)
    p[:, m["s1"][0]] = np.repeat(a, n2)
    p[:, m["s2"][0]] = np.tile(b, n1)
    return p


def _map_inputs(name, n1, n2, rng):
    """Parameters and jittered initial states, as the benchmark draws them."""
    m = MODELS[name]
    p = _grid(m, n1, n2)
    if name == "lorenz96":  # x0 = F + N(0, 0.01^2)
        return p, p[:, :1] + 0.01 * rng.standard_normal((n1 * n2, 40))
    return p, np.asarray(m["x0"]) + rng.uniform(-1e-3, 1e-3, (n1 * n2, len(m["x0"])))


def _compat_inputs(c, rng):
    return _map_inputs(c["model"], c["n1"], c["n2"], rng)


def _trajectory_inputs(c, rng):
    m = MODELS[c["model"]]
    P = c["P"]
    p = np.tile(np.asarray(m["base"]), (P, 1))
    for i, lo, hi in (m["s1"], m["s2"]):
        p[:, i] = rng.uniform(lo, hi, P)
    return p, np.asarray(m["x0"]) + rng.uniform(-1e-3, 1e-3, (P, len(m["x0"])))


def _net_inputs(c, rng):
    """Weights (He-style uniform), parameter points, and targets shaped like a
    Lorenz map's spectra with the regime score as the fourth output."""
    E, W, rows = c["E"], c["W"], c["rows"]
    nets = []
    for _ in range(E):
        parts = []
        for fan_in, cols in ((16, W), (W, W), (W, W), (W, 16)):
            w = math.sqrt(6.0 / fan_in) * rng.uniform(-1, 1, (fan_in, cols))
            if cols == 16:
                w *= 0.5
                w[:, 4:] = 0.0
            parts += [w.ravel(), np.zeros(cols)]
        nets.append(np.concatenate(parts))
    weights = np.stack(nets).astype(np.float32)
    xy = np.stack([rng.uniform(DOMAIN[0], DOMAIN[1], rows),
                   rng.uniform(DOMAIN[2], DOMAIN[3], rows)], 1)
    s = np.tanh((xy[:, 1] - 30.0) / 20.0)
    y = np.stack([0.9 * s, 0.05 * np.sin(xy[:, 0]), -(xy[:, 0] + 11.0 / 3.0) - 0.9 * s,
                  np.tanh((0.9 * s - 0.01) / 0.05)], 1)
    return weights, xy, y


def _net(c, weights, y):
    net = MLPEnsemble(ensemble=c["E"], width=c["W"], outputs=4, seed=1)
    net.set_domain(*DOMAIN)
    net.set_target_scale(y.mean(0), y.std(0))
    net.set_params(weights)
    return net


def _out(P, k):
    return (torch.zeros((P, k), dtype=torch.float64, device="cuda"),
            torch.full((P,), -1, dtype=torch.int32, device="cuda"))


def prepare(case, seed):
    c = case
    rng = np.random.default_rng(seed)
    if c["kind"] in ("map", "host"):
        p, x = _map_inputs(c["model"], c["n1"], c["n2"], rng)
        kw = dict(schedule=c["schedule"], block=c["block"], variant=c["variant"]) \
            if c["kind"] == "map" else {}
        sweep = cl.Sweep(model=c["model"], method="var", integrator=c["integrator"],
                         precision=c["precision"], rtol=c["rtol"], atol=c["rtol"],
                         gs="mgs" if c["model"] == "lorenz96" else "cgs",
                         h=1e-2 if c["model"] == "lorenz96" else 1e-3, t_transient=c["t_tr"],
                         t_avg=c["t_avg"], dt_renorm=c["dt"], **kw)
        if c["kind"] == "host":
            return dict(kind="host", sweep=sweep, p=p, x=x)
        spec, status = _out(p.shape[0], sweep.k)
        return dict(kind="map", sweep=sweep, p=torch.from_numpy(p).cuda(),
                    x=torch.from_numpy(x).cuda(), spec=spec, status=status)
    if c["kind"] == "batch":
        parts = []
        for name in ("hyper_rossler", "lorenz", "chua"):
            p, x = _map_inputs(name, c["n"], c["n"], rng)
            sweep = cl.Sweep(model=name, method="var", integrator="dopri5", precision="fp32",
                             rtol=1e-6, atol=1e-6, h=1e-2, t_transient=c["t_tr"],
                             t_avg=c["t_hi"], dt_renorm=1.0, block=128,
                             schedule="split_persistent" if name == "hyper_rossler" else "auto")
            t = rng.uniform(c["t_lo"], c["t_hi"], p.shape[0])
            spec, status = _out(p.shape[0], sweep.k)
            parts.append((sweep, torch.from_numpy(p).cuda(), torch.from_numpy(x).cuda(), spec,
                          status, None, torch.from_numpy(t).cuda()))
        return dict(kind="batch", parts=parts, graph=cl.BatchGraph(parts))
    if c["kind"] == "compat":
        p, x = _compat_inputs(c, rng)
        P = p.shape[0]
        return dict(kind="compat", case=c, P=P, p=torch.from_numpy(p).cuda(),
                    x0=torch.from_numpy(x).cuda(), x=torch.empty((P, 3), dtype=torch.float64,
                                                                  device="cuda"),
                    lyap=torch.empty((P, 3), dtype=torch.float64, device="cuda"),
                    close=torch.empty((P, 9), dtype=torch.float64, device="cuda"))
    if c["kind"] == "trajectory":
        p, x = _trajectory_inputs(c, rng)
        sweep = cl.Sweep(model=c["model"], integrator=c["integrator"], precision=c["precision"],
                         rtol=c["rtol"], atol=c["rtol"], h=1e-3, t_avg=1.0, dt_renorm=1.0)
        return dict(kind="trajectory", sweep=sweep, p=torch.from_numpy(p).cuda(),
                    x=torch.from_numpy(x).cuda(), nsteps=c["nsteps"])
    weights, xy, y = _net_inputs(c, rng)
    state = dict(kind=c["kind"], net=_net(c, weights, y), xy=torch.from_numpy(xy).cuda())
    if c["kind"] == "train":
        state.update(y=torch.from_numpy(y).cuda(), steps=c["steps"], batch=c["batch"])
    return state


def run(state):
    s = state
    if s["kind"] == "host":
        return s["sweep"].run_host(s["p"], s["x"])
    if s["kind"] == "map":
        s["sweep"].run(s["p"], s["x"], s["spec"], s["status"])
        return s["spec"], s["status"]
    if s["kind"] == "batch":
        s["graph"].launch()
        return [(part[3], part[4]) for part in s["parts"]]
    if s["kind"] == "compat":
        c = s["case"]
        s["x"].copy_(s["x0"])  # the launcher advances the states in place
        s["lyap"].zero_()      # and adds to the exponents
        cl.cuda_lyapunov(s["P"], c["method"] == "qr", c["method"] == "var", s["x"],
                         None if c["method"] == "qr" else s["close"], 3, c["model"], s["p"],
                         s["p"].shape[1], 1e-7, c["h"], s["lyap"], 3, c["t_skip"], c["t_clp"],
                         c["t_calc"], c["t_norm"] / c["h"])
        return (s["lyap"], s["x"]) if c["method"] == "qr" else (s["lyap"], s["x"], s["close"])
    if s["kind"] == "trajectory":
        return s["sweep"].trajectory(s["p"], s["x"], s["nsteps"])
    if s["kind"] == "train":
        loss = s["net"].train(s["xy"], s["y"], s["steps"], s["batch"], 1e-3, 3)
        return s["net"].get_params(), loss
    return s["net"].predict(s["xy"])


# -------------------------------------------------------------------- work
STAGES = {"dopri5": (6, 26), "dverk65": (8, 39)}  # new stages, tableau coefficients


def _step_flops(model, integrator, n):
    """The state and its n tangent vectors, one attempted step."""
    S, C = STAGES[integrator]
    f, jv = MODELS[model]["flops"]
    return S * (f + n * jv) + 2 * C * n * (1 + n)


def _state_flops(model, integrator, n):
    S, C = STAGES[integrator]
    return S * MODELS[model]["flops"][0] + 2 * C * n


def _rate(model, integrator, rtol):
    return MODELS[model]["rate"][0 if integrator == "dopri5" and rtol > 1e-9 else 1] \
        * (1.0 if rtol < 1e-9 or integrator == "dopri5" else 0.25)


def work(case):
    c = case
    if c["kind"] in ("map", "host"):
        m = MODELS[c["model"]]
        n = 40 if c["model"] == "lorenz96" else len(m["x0"])
        P = c["n1"] * c["n2"]
        r = _rate(c["model"], c["integrator"], c["rtol"])
        flops = P * r * (c["t_tr"] * _state_flops(c["model"], c["integrator"], n)
                         + c["t_avg"] * _step_flops(c["model"], c["integrator"], n))
        return {"bytes": P * (8 * (len(m["base"]) + 2 * n) + 4), "flops": flops}
    if c["kind"] == "batch":
        P, flops, size = c["n"] * c["n"], 0.0, 0
        for name in ("hyper_rossler", "lorenz", "chua"):
            m = MODELS[name]
            n = len(m["x0"])
            flops += P * m["rate"][0] * (c["t_tr"] * _state_flops(name, "dopri5", n)
                                         + 0.5 * (c["t_lo"] + c["t_hi"])
                                         * _step_flops(name, "dopri5", n))
            size += P * (8 * (len(m["base"]) + 2 * n + 1) + 4)
        return {"bytes": size, "flops": flops}
    if c["kind"] == "compat":
        P = c["n1"] * c["n2"]
        S, C = 8, 33  # fixed-step DVERK: no error estimate
        f, jv = MODELS[c["model"]]["flops"]
        state = S * f + 2 * C * 3
        rows = 3 * (S * (f if c["method"] == "fd" else jv) + 2 * C * 3)
        steps = (c["t_skip"] / c["h"], (c["t_clp"] + c["t_calc"]) / c["h"])
        close = 0 if c["method"] == "qr" else 9
        return {"bytes": P * 8 * (len(MODELS[c["model"]]["base"]) + 9 + close),
                "flops": P * (steps[0] * state + steps[1] * (state + rows))}
    if c["kind"] == "trajectory":
        return {"bytes": c["P"] * (8 * (6 + 5 * c["nsteps"]) + 4),
                "flops": c["P"] * c["nsteps"] * _state_flops(c["model"], c["integrator"], 3)}
    W, E = c["W"], c["E"]
    weights = 16 * W + 2 * W * W + 16 * W
    forward = 2.0 * E * weights
    if c["kind"] == "train":  # forward, gradients of activations and of weights, Adam
        rows = min(c["batch"], c["rows"])
        return {"bytes": c["rows"] * 48 + E * (weights + 3 * W + 16) * 4,
                "flops": c["steps"] * (3.0 * rows * forward + 10.0 * E * weights)}
    return {"bytes": c["rows"] * (16 + 2 * 16) + E * weights * 4, "flops": c["rows"] * forward}


# ------------------------------------------------------- 64-bit references
def _f(model, x, p):
    a, b, c = x[..., 0], x[..., 1], x[..., 2]
    q = [p[:, i].reshape(-1, *([1] * (x.dim() - 2))) for i in range(p.shape[1])]
    if model == "lorenz":
        return torch.stack([q[0] * (b - a), a * (q[1] - c) - b, a * b - q[2] * c], -1)
    if model == "rossler":
        return torch.stack([-b - c, a + q[0] * b, q[1] + c * (a - q[2])], -1)
    return torch.stack([b, -q[0] * b - a * c + a, -q[1] * c + a * a], -1)  # shimizu


def _jac(model, x, p):
    a, b, c = x[:, 0], x[:, 1], x[:, 2]
    o, l = torch.zeros_like(a), torch.ones_like(a)
    if model == "lorenz":
        rows = [-p[:, 0], p[:, 0], o, p[:, 1] - c, -l, -a, b, a, -p[:, 2]]
    elif model == "rossler":
        rows = [o, -l, -l, l, p[:, 0], o, c, o, a - p[:, 2]]
    else:
        rows = [o, l, o, l - c, -p[:, 0], -a, 2 * a, o, -p[:, 1]]
    return torch.stack(rows, 1).view(-1, 3, 3)


DVERK_A = [[], [1 / 6], [4 / 75, 16 / 75], [5 / 6, -8 / 3, 5 / 2],
           [-165 / 64, 55 / 6, -425 / 64, 85 / 96],
           [12 / 5, -8, 4015 / 612, -11 / 36, 88 / 255],
           [-8263 / 15000, 124 / 75, -643 / 680, -81 / 250, 2484 / 10625],
           [3501 / 1720, -300 / 43, 297275 / 52632, -319 / 2322, 24068 / 84065, 0, 3850 / 26703]]
DVERK_B = [3 / 40, 0, 875 / 2244, 23 / 72, 264 / 1955, 0, 125 / 11592, 43 / 616]
DOPRI_A = [[], [1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
           [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
           [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656]]
DOPRI_B = [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]
DOPRI_E = [71 / 57600, 0, -71 / 16695, 71 / 1920, -17253 / 339200, 22 / 525, -1 / 40]


def _comb(coef, ks):
    return sum(c * k for c, k in zip(coef, ks) if c)


def _rk(f, y, h):
    """One DVERK step of y' = f(y)."""
    ks = []
    for a in DVERK_A:
        ks.append(f(y + h * _comb(a, ks) if a else y))
    return y + h * _comb(DVERK_B, ks)


def _orth(v):
    """Classical Gram-Schmidt of the rows of v; the unit rows and the lengths."""
    out, r = [], []
    for i in range(v.shape[1]):
        w = v[:, i]
        for u in out:
            w = w - (u * v[:, i]).sum(1, keepdim=True) * u
        n = w.norm(dim=1, keepdim=True)
        out.append(w / n)
        r.append(n[:, 0])
    return torch.stack(out, 1), torch.stack(r, 1)


def _count(T, h):
    """Passes of `for (t = 0; t < T; t += h)`."""
    n, t = 0, 0.0
    while t < T:
        n, t = n + 1, t + h
    return n


def _exact_compat(c, seed):
    p, x = (torch.from_numpy(a).cuda() for a in _compat_inputs(c, np.random.default_rng(seed)))
    m, h, eps = c["model"], c["h"], 1e-7
    P, calc = p.shape[0], _count(c["t_calc"], c["h"])
    for _ in range(_count(c["t_skip"], h)):
        x = _rk(lambda y: _f(m, y, p), x, h)
    v = torch.eye(3, dtype=torch.float64, device="cuda").repeat(P, 1, 1)
    lyap = torch.zeros((P, 3), dtype=torch.float64, device="cuda")
    if c["method"] == "fd":  # perturbed copies, integrated by the flow itself
        s = x[:, None] + eps * v

        def advance(x, s):
            y = _rk(lambda y: _f(m, y, p), torch.cat([x[:, None], s], 1), h)
            return y[:, 0], y[:, 1:]

        for _ in range(_count(c["t_clp"], h)):
            x, s = advance(x, s)
            s = x[:, None] + eps * _orth(s - x[:, None])[0]
        for i in range(calc):
            x, s = advance(x, s)
            if (i + 1) % round(c["t_norm"] / h) == 0:
                u, r = _orth(s - x[:, None])
                lyap += (r / eps).log()
                s = x[:, None] + eps * u
        return lyap / c["t_calc"], x, s
    for i in range((_count(c["t_clp"], h) if c["method"] == "var" else 0) + calc):
        align = c["method"] == "var" and i < _count(c["t_clp"], h)
        xn = _rk(lambda y: _f(m, y, p), x, h)
        # VAR freezes the state over its step; QR's state has already moved
        J = _jac(m, x if c["method"] == "var" else xn, p).transpose(1, 2)
        v = _rk(lambda y: y @ J, v, h)
        x = xn
        j = i - _count(c["t_clp"], h) if c["method"] == "var" else i
        if align or c["method"] == "qr" or (j + 1) % round(c["t_norm"] / h) == 0:
            v, r = _orth(v)
            if not align:
                lyap += r.log()
    if c["method"] == "qr":
        return lyap / c["t_calc"], x
    return lyap / c["t_calc"], x, eps * v


def _exact_host(c, seed):
    """The joint state and tangent equations at a small fixed step."""
    p, x = _map_inputs(c["model"], c["n1"], c["n2"], np.random.default_rng(seed))
    p, x = torch.from_numpy(p).cuda(), torch.from_numpy(x).cuda()
    m, P, h = c["model"], p.shape[0], 2.5e-3

    def joint(y):
        return torch.cat([_f(m, y[:, :1], p), y[:, 1:] @ _jac(m, y[:, 0], p).transpose(1, 2)], 1)

    for _ in range(round(c["t_tr"] / h)):
        x = _rk(lambda y: _f(m, y, p), x, h)
    y = torch.cat([x[:, None], torch.eye(3, dtype=torch.float64, device="cuda").repeat(P, 1, 1)], 1)
    s = torch.zeros((P, 3), dtype=torch.float64, device="cuda")
    for i in range(round(c["t_avg"] / h)):
        y = _rk(joint, y, h)
        if i % 10 == 9:
            v, r = _orth(y[:, 1:])
            s += r.log()
            y = torch.cat([y[:, :1], v], 1)
    return s / c["t_avg"], None


def _exact_trajectory(c, seed):
    """Dormand-Prince 5(4) with the library's documented step control."""
    if c["integrator"] != "dopri5" or c["precision"] != "fp64":
        return None
    p, x = (torch.from_numpy(a).cuda() for a in _trajectory_inputs(c, np.random.default_rng(seed)))
    P, n, tol = p.shape[0], c["nsteps"], c["rtol"]
    new = dict(dtype=torch.float64, device="cuda")
    t_out, h_out = torch.zeros((P, n), **new), torch.zeros((P, n), **new)
    x_out = torch.zeros((P, n, 3), **new)
    t, h = torch.zeros(P, **new), torch.full((P,), 1e-3, **new)
    old = torch.full((P,), 1e-4, **new)
    rejected = torch.zeros(P, dtype=torch.bool, device="cuda")
    rec = torch.zeros(P, dtype=torch.int64, device="cuda")
    k1 = _f(c["model"], x, p)
    rows = torch.arange(P, device="cuda")
    for _ in range(4 * n):
        ks = [k1]
        for a in DOPRI_A[1:]:
            ks.append(_f(c["model"], x + h[:, None] * _comb(a, ks), p))
        y = x + h[:, None] * _comb(DOPRI_B, ks)
        ks.append(_f(c["model"], y, p))
        e = h[:, None] * _comb(DOPRI_E, ks) / (tol + tol * torch.maximum(x.abs(), y.abs()))
        err = e.square().mean(1).sqrt()
        live = rec < n
        ok = (err <= 1.0) & live
        fac = (err ** 0.17 / old ** 0.04 / 0.9).clamp(0.1, 5.0)
        hn = h / fac
        hn = torch.where(rejected, torch.minimum(hn, h), hn)
        ht = torch.where(ok, hn, h / (err ** 0.17 / 0.9).clamp(max=5.0))
        t = torch.where(ok, t + h, t)
        x = torch.where(ok[:, None], y, x)
        k1 = torch.where(ok[:, None], ks[-1], k1)
        old = torch.where(ok, err.clamp(min=1e-4), old)
        rejected = torch.where(live, ~ok, rejected)
        h = torch.where(live, ht, h)
        r, q = rows[ok], rec[ok]
        t_out[r, q], h_out[r, q], x_out[r, q] = t[ok], h[ok], x[ok]
        rec = rec + ok
        if int(rec.min()) >= n:
            break
    return t_out, h_out, x_out, None


def _features(xy):
    u = (xy[:, 0] - DOMAIN[0]) / (DOMAIN[1] - DOMAIN[0])
    v = (xy[:, 1] - DOMAIN[2]) / (DOMAIN[3] - DOMAIN[2])
    cols = []
    for j in range(1, 5):
        for w in (u, v):
            cols += [torch.sin(math.pi * j * w), torch.cos(math.pi * j * w)]
    return torch.stack(cols, 1)


def _layers(flat, W):
    out, o = [], 0
    for r, c in ((16, W), (W, W), (W, W), (W, 16)):
        out.append((flat[o:o + r * c].view(r, c), flat[o + r * c:o + r * c + c]))
        o += r * c + c
    return out


def _forward(flat, W, feats):
    h = feats
    for i, (w, b) in enumerate(_layers(flat, W)):
        h = h @ w + b
        if i < 3:
            h = h * torch.sigmoid(h)
    return h[:, :4]


def _exact_predict(c, seed):
    weights, xy, y = _net_inputs(c, np.random.default_rng(seed))
    mean = torch.from_numpy(y.mean(0)).cuda()
    std = torch.from_numpy(y.std(0)).cuda()
    out = [[], []]
    for o in range(0, c["rows"], 1 << 17):
        feats = _features(torch.from_numpy(xy[o:o + (1 << 17)]).cuda())
        ys = torch.stack([_forward(torch.from_numpy(w.astype(np.float64)).cuda(), c["W"], feats)
                          for w in weights]) * std + mean
        out[0].append(ys.mean(0))
        out[1].append(ys.std(0, correction=0))
    return torch.cat(out[0]), torch.cat(out[1])


def _exact_train(c, seed):
    """Adam on the mean squared error of the standardised targets, minibatches
    from the library's seeded shuffles (seed 3)."""
    weights, xy, y = _net_inputs(c, np.random.default_rng(seed))
    feats = _features(torch.from_numpy(xy).cuda())
    target = torch.from_numpy((y - y.mean(0)) / y.std(0)).cuda()
    N, B = c["rows"], min(c["batch"], c["rows"])
    p = torch.from_numpy(weights.astype(np.float64)).cuda().requires_grad_(True)
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    mask = (1 << 64) - 1
    st = (3 * 0x9E3779B97F4A7C15 + 1) & mask
    perm, pos, loss = list(range(N)), N, None
    for t in range(1, c["steps"] + 1):
        idx = []
        while len(idx) < B:
            if pos >= N:
                for i in range(N - 1, 0, -1):
                    st = (st ^ (st << 13)) & mask
                    st ^= st >> 7
                    st = (st ^ (st << 17)) & mask
                    j = st % (i + 1)
                    perm[i], perm[j] = perm[j], perm[i]
                pos = 0
            take = perm[pos:pos + B - len(idx)]
            idx += take
            pos += len(take)
        idx = torch.tensor(idx, device="cuda")
        loss = torch.stack([(_forward(p[z], c["W"], feats[idx]) - target[idx]).square().mean()
                            for z in range(c["E"])])
        g, = torch.autograd.grad(loss.sum(), p)
        with torch.no_grad():
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            p -= 1e-3 * (m / (1 - 0.9 ** t)) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8)
    return p.detach(), loss.detach()


def exact(case, seed):
    c = case
    if c["kind"] == "host":
        return _exact_host(c, seed)
    if c["kind"] == "compat":
        return _exact_compat(c, seed)
    if c["kind"] == "trajectory":
        return _exact_trajectory(c, seed)
    if c["kind"] == "predict":
        return _exact_predict(c, seed)
    if c["kind"] == "train":
        return _exact_train(c, seed)
    return None  # the other horizons take minutes in plain torch
