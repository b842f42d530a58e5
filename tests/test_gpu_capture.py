"""Stream captures: a batch captured at its handles' first use, and sweeps on
other streams while a capture is open."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KW = dict(method="var", precision="fp64", integrator="dopri5", rtol=1e-8, atol=1e-8, h=1e-3,
          t_transient=2.0, t_avg=4.0, dt_renorm=1.0, schedule="persistent")
MODELS = {"lorenz": ([10.0, 15.0, 8.0 / 3.0], [1.0, 1.0, 1.0]),
          "rossler": ([0.2, 0.2, 4.0], [1.0, 1.0, 0.0]),
          "hyper_rossler": ([0.25, 0.05], [-10.0, -6.0, 0.0, 10.0])}


def _part(lib, torch, model, P):
    pb, xb = MODELS[model]
    rng = np.random.default_rng(P)
    p = torch.from_numpy(np.array(pb) * (1 + 0.01 * rng.uniform(-1, 1, (P, len(pb))))).cuda()
    x = torch.from_numpy(np.array(xb) + rng.uniform(-1e-3, 1e-3, (P, len(xb)))).cuda()
    spec = torch.zeros((P, len(xb)), dtype=torch.float64, device="cuda")
    status = torch.full((P,), -1, dtype=torch.int32, device="cuda")
    return lib.Sweep(model=model, **KW), p, x, spec, status, None, None


def test_batch_captured_at_first_use(lib):
    """The batch's further streams and events are made inside the capture."""
    import torch
    from chaos_oneapi_b200.sweep import run_batch
    parts = [_part(lib, torch, m, P) for m, P in (("lorenz", 500), ("rossler", 400),
                                                  ("hyper_rossler", 300))]
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        run_batch(parts)
    g.replay()
    torch.cuda.synchronize()
    captured = [q[3].clone() for q in parts]
    for q in parts:
        assert (q[4] == 0).all()
        q[3].zero_()
    run_batch(parts)
    torch.cuda.synchronize()
    for q, want in zip(parts, captured):
        assert torch.equal(q[3], want)  # fewer points than lanes: the same warps
        q[0].close()


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
@pytest.mark.parametrize("own_thread", [True, False])
def test_sweep_beside_an_open_capture(lib, mode, own_thread):
    """A sweep of two launches takes its buffers from a pool, which must not end
    a capture that is open on another stream."""
    import torch
    P = 60_001  # above 1.5 waves
    sw, p, x, spec, status, _, _ = _part(lib, torch, "lorenz", P)
    z = torch.zeros(8, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    errors = []

    def run():
        try:
            sw.run(p, x, spec, status, stream=stream.cuda_stream)
        except Exception as e:  # reported after the capture has ended
            errors.append(e)

    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode=mode):
        z.add_(1)
        if own_thread:
            run()
        else:
            t = threading.Thread(target=run)
            t.start()
            t.join()
        z.add_(1)
    g.replay()
    torch.cuda.synchronize()
    assert not errors
    assert (z == 2).all() and (status == 0).all()
    sw.close()


def test_sweep_of_own_times_captured_after_a_run(lib):
    """A run makes what a later capture of the same call needs, also where the
    run itself takes two launches and the captured one one."""
    import torch
    P = 60_001
    sw, p, x, spec, status, _, _ = _part(lib, torch, "lorenz", P)
    t_avg = torch.linspace(0.5, 4.0, P, dtype=torch.float64, device="cuda")
    sw.run(p, x, spec, status, t_avg=t_avg)
    torch.cuda.synchronize()
    assert sw.launches() == 6
    spec.zero_()
    status.fill_(-1)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        sw.run(p, x, spec, status, t_avg=t_avg)
    assert sw.launches() == 5
    g.replay()
    torch.cuda.synchronize()
    assert (status == 0).all()
    # the exponents add up to the trace -(sigma + 1 + beta) on every cell, also
    # beside a separatrix, where single exponents depend on the grouping; to the
    # integration error, some 1e3 rtol
    assert (spec.sum(1) + p[:, 0] + 1 + p[:, 2]).abs().max() < 1e3 * KW["rtol"]
    sw.close()
