"""Sweeps in two launches against the one-launch form of the same points and
against the exact exponents: chaotic FP32 maps, the 4-dimensional model, the
96-register build, an alignment phase, and points that run out of steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MODELS = {
    "lorenz": (lambda u, v: [5 + 15 * u, 200 * v, 8 / 3 + 0 * u], [1.0, 1.0, 1.0]),
    "rossler": (lambda u, v: [0.1 + 0.25 * u, 0.2 + 0 * u, 2 + 10 * v], [1.0, 1.0, 0.0]),
    "hyper_rossler": (lambda u, v: [0.2 + 0.08 * u, 0.03 + 0.03 * v], [-10.0, -6.0, 0.0, 10.0]),
}


class Map:
    """P points of a model's map, in no spatial order."""

    def __init__(self, lib, torch, model, P):
        rng = np.random.default_rng(P)
        f, x0 = MODELS[model]
        u, v = rng.uniform(0, 1, (2, P))
        self.lib, self.torch, self.model, self.n = lib, torch, model, len(x0)
        self.p = torch.from_numpy(np.stack(f(u, v), 1)).cuda()
        self.x = torch.from_numpy(np.array(x0) + rng.uniform(-1e-3, 1e-3, (P, len(x0)))).cuda()

    def run(self, capture=False, **kw):
        torch, P = self.torch, self.p.shape[0]
        sw = self.lib.Sweep(model=self.model, method="var", h=1e-3, dt_renorm=1.0,
                            schedule="persistent", **kw)
        out = torch.zeros((P, self.n), dtype=torch.float64, device="cuda")
        st = torch.full((P,), -1, dtype=torch.int32, device="cuda")
        steps = torch.zeros(P, dtype=torch.int64, device="cuda")
        if capture:  # a captured sweep takes one launch
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                sw.run(self.p, self.x, out, st, steps)
            g.replay()
        else:
            sw.run(self.p, self.x, out, st, steps)
        torch.cuda.synchronize()
        assert sw.launches() == (1 if capture else 6)
        sw.close()
        return out.cpu().numpy(), st.cpu().numpy(), steps.cpu().numpy()


# points: 1.6 waves of 512 (variant 1: 640) FP32 or 256 FP64 points on 148 SMs
@pytest.mark.parametrize("model,P,times,kw", [
    ("rossler", 121_243, (30, 100, 0), dict(precision="fp32", integrator="dopri5")),
    ("rossler", 151_553, (30, 100, 0), dict(precision="fp32", integrator="dopri5", variant=1)),
    ("rossler", 121_243, (30, 100, 20), dict(precision="fp32", integrator="dverk65")),
    ("lorenz", 121_243, (10, 40, 0), dict(precision="fp32", integrator="dopri5")),
    ("hyper_rossler", 121_243, (20, 60, 0), dict(precision="fp32", integrator="dopri5")),
    ("hyper_rossler", 60_623, (20, 60, 5), dict(precision="fp64", integrator="dverk65")),
], ids=lambda v: "-".join(map(str, v.values())) if isinstance(v, dict) else None)
def test_as_close_to_the_exact_exponents(lib, model, P, times, kw):
    """On cells whose exponents do not depend on the tolerance, the errors of the
    two forms have the same distribution: no quantile of the two-launch form's is
    more than a quarter larger (the spread of a 1 % quantile over thousands of
    cells is about a tenth)."""
    import torch
    m = Map(lib, torch, model, P)
    t = dict(t_transient=times[0], t_avg=times[1], t_align=times[2])
    rtol = 1e-6 if kw["precision"] == "fp32" else 1e-8
    two, st2, _ = m.run(rtol=rtol, atol=rtol, **t, **kw)
    one, st1, _ = m.run(capture=True, rtol=rtol, atol=rtol, **t, **kw)
    tight = dict(precision="fp64", integrator="dverk65", **t)
    ref, st, _ = m.run(capture=True, rtol=1e-12, atol=1e-12, **tight)
    ref2, _, _ = m.run(capture=True, rtol=1e-11, atol=1e-11, **tight)
    assert np.mean(st1 != st2) < 1e-3
    ok = (st == 0) & (st1 == 0) & (st2 == 0)
    regular = ok & (np.abs(ref - ref2).max(1) < 1e-6)
    assert regular.sum() > 5000
    e2, e1 = (np.abs(a - ref)[regular].max(1) for a in (two, one))
    for q in (0.5, 0.9, 0.99):
        assert np.quantile(e2, q) < 1.25 * np.quantile(e1, q), q


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_step_budget(lib, precision):
    """Every point runs out of steps: some in the transient, the others in the
    averaging phase, all with the same status and count as in one launch."""
    import torch
    m = Map(lib, torch, "lorenz", 121_243)
    kw = dict(precision=precision, integrator="dopri5", rtol=1e-6, atol=1e-6, t_transient=3.0,
              t_avg=500.0)
    _, _, transient = m.run(**dict(kw, t_avg=1e-3))
    budget = int(np.median(transient))
    out, st, steps = m.run(max_steps=budget, **kw)
    assert (transient > budget).sum() > 1000 and (transient < budget).sum() > 1000
    assert (st == 3).all() and (steps == budget).all() and np.isnan(out).all()
