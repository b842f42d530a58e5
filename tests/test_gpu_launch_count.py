"""chaos_lyap_get_launches: how many kernels a run enqueued, which tells the form
it took (bench.py reports it)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KW = dict(method="var", rtol=1e-6, atol=1e-6, h=1e-3, t_avg=0.2, dt_renorm=0.1)


def _arrays(torch, dim, p0, P):
    p = torch.tensor(p0, dtype=torch.float64, device="cuda").repeat(P, 1)
    x = torch.full((P, dim), 1.0, dtype=torch.float64, device="cuda")
    x[:, 0] += torch.linspace(0, 1e-3, P, dtype=torch.float64, device="cuda")
    return p, x, torch.zeros((P, dim), dtype=torch.float64, device="cuda")


# 148 SMs hold 256 FP64 or 512 FP32 points each (16 of Lorenz-96); two launches
# from 1.5 (1) to 32 times that
@pytest.mark.parametrize("kw,P,kernels", [
    (dict(precision="fp32", t_transient=0.1), 113_664, 1),
    (dict(precision="fp32", t_transient=0.1), 113_665, 6),
    (dict(precision="fp32", t_transient=0.0), 113_665, 1),
    (dict(precision="fp32", t_transient=0.1, schedule="split"), 113_665, 1),
    (dict(precision="fp64", t_transient=0.1), 56_832, 1),
    (dict(precision="fp64", t_transient=0.1), 56_833, 6),
    (dict(precision="fp32", t_transient=0.1, model="lorenz96"), 2368, 1),
    (dict(precision="fp32", t_transient=0.1, model="lorenz96"), 2369, 6),
    (dict(precision="compat", integrator="dverk"), 500, 1),
], ids=str)
def test_sweeps(lib, kw, P, kernels):
    import torch
    cfg = dict(dict(KW, model="lorenz", integrator="dopri5"), **kw)
    dim, p0 = (40, [8.0, 1.0]) if cfg["model"] == "lorenz96" else (3, [10.0, 15.0, 8.0 / 3.0])
    sw = lib.Sweep(**cfg)
    assert sw.launches() == 0
    sw.run(*_arrays(torch, dim, p0, P))
    assert sw.launches() == kernels
    sw.sync()
    sw.close()


def test_own_times_and_batches(lib):
    import torch
    from chaos_oneapi_b200.sweep import run_batch
    cfg = dict(KW, model="lorenz", integrator="dopri5", precision="fp32")
    parts = []
    for P, own in ((300, True), (0, False), (200, False)):
        p, x, out = _arrays(torch, 3, [10.0, 15.0, 8.0 / 3.0], P)
        ta = torch.full((P,), 0.2, dtype=torch.float64, device="cuda") if own else None
        parts.append((lib.Sweep(**cfg), p, x, out, None, None, ta))
    sw, p, x, out, _, _, ta = parts[0]
    sw.run(p, x, out, t_avg=ta)
    assert sw.launches() == 5
    run_batch(parts)
    assert sw.launches() == 6 and parts[2][0].launches() == 0
    g = lib.BatchGraph(parts)
    assert sw.launches() == 6
    g.launch()
    torch.cuda.synchronize()
    g.close()
    for q in parts:
        q[0].close()
