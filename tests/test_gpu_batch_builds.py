"""FP32 batches of points with averaging times of their own: the launch forms
they run in (a build of up to 168 registers in a few waves, on two blocks per SM in
a batch of one segment; the sweeps' own build from three waves on) against sweeps
of the same points."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# regular cells: the exponents do not depend on when a warp renormalises
MODELS = {"shimizu": ([0.8, 2.5], [0.1, 0.05, 0.02]), "lorenz": ([10.0, 12.0, 8.0 / 3.0], [1.0, 1.0, 1.0]),
          "rossler": ([0.2, 0.2, 2.5], [1.0, 1.0, 0.0]),
          "chua": ([5.0, 20.0, -8.0 / 7.0, -5.0 / 7.0], [0.1, 0.0, 0.0]),
          "hyper_rossler": ([0.25, 0.05], [-10.0, -6.0, 0.0, 10.0])}
KW = dict(method="var", precision="fp32", rtol=1e-6, atol=1e-6, h=1e-3, t_transient=1.0, t_avg=1.0,
          dt_renorm=1.0)


def _inputs(model, P, block, integrator):
    import chaos_oneapi_b200 as lib
    import torch
    pb, xb = MODELS[model]
    rng = np.random.default_rng(P)
    p = np.array(pb) * (1 + 0.02 * rng.uniform(-1, 1, (P, len(pb))))
    x = np.array(xb) + rng.uniform(-1e-3, 1e-3, (P, len(xb)))
    x[::997, 0] = 2e4  # outside the escape radius
    return (lib.Sweep(model=model, block=block, integrator=integrator, schedule="persistent", **KW),
            *(torch.from_numpy(a).cuda() for a in (p, x, rng.uniform(0.5, 2.0, P))))


@pytest.mark.parametrize("integrator", ["dopri5", "dverk65"])
@pytest.mark.parametrize("spec", [
    (("lorenz", 3000),), (("rossler", 50_001),), (("hyper_rossler", 50_001),),  # two blocks per SM
    (("shimizu", 120_001),), (("lorenz", 240_001),),                           # own build last
    (("chua", 40_001), ("lorenz", 257), ("hyper_rossler", 30_001), ("shimizu", 0)),
    (("chua", 1001), ("rossler", 997))], ids=lambda s: "-".join(f"{m}{n}" for m, n in s))
@pytest.mark.parametrize("block", [128, 64])
def test_batch_matches_sweeps(lib, spec, integrator, block):
    import torch
    from chaos_oneapi_b200.sweep import run_batch
    parts = []
    for model, P in spec:
        sw, p, x, ta = _inputs(model, P, block, integrator)
        out = torch.full((P, x.shape[1]), 7.0, dtype=torch.float64, device="cuda")
        parts.append((sw, p, x, out, torch.full((P,), -1, dtype=torch.int32, device="cuda"),
                      torch.zeros(P, dtype=torch.int64, device="cuda"), ta))
    run_batch(parts)
    torch.cuda.synchronize()
    for sw, p, x, out, status, steps, ta in parts:
        P = p.shape[0]
        if not P:
            continue
        tight = dict(KW, model=sw.cfg.model, precision="fp64", integrator="dverk65", rtol=1e-11,
                     atol=1e-11, schedule="persistent")
        ref = lib.Sweep(**tight)
        want, own = torch.zeros_like(out), torch.zeros_like(out)
        wst, ost = torch.zeros_like(status), torch.zeros_like(status)
        sw.run(p, x, own, ost, t_avg=ta)
        ref.run(p, x, want, wst, t_avg=ta)
        torch.cuda.synchronize()
        assert torch.equal(status, ost) and torch.equal(status, wst)
        ok = status == 0
        assert int((~ok).sum()) == (P + 996) // 997 and torch.isnan(out[~ok]).all()
        assert (steps[ok] > 0).all()
        # the same method on the same points, renormalised at other times: no
        # further from the exact exponents than the sweep, up to the spread of a
        # root mean square over thousands of cells
        got, sweep = ((a[ok] - want[ok]).pow(2).mean().sqrt() for a in (out, own))
        assert got < 1.25 * sweep, (sw.cfg.model, float(got), float(sweep))
        sw.close()
        ref.close()
