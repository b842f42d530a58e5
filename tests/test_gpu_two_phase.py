"""Sweeps in two launches (all transients, then the averaging phases, longest
expected first) against the one-launch form of the same points: the same
statuses, the same transients, and spectra that differ only by when the warps
renormalised."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RTOL = 1e-8


def _inputs(P, seed=3):
    """Lorenz below the onset of chaos (rho < 20); every 97th point starts outside
    the escape radius, every 101st has a NaN parameter."""
    rng = np.random.default_rng(seed)
    p = np.stack([rng.uniform(5, 20, P), rng.uniform(1.5, 20, P), np.full(P, 8.0 / 3.0)], 1)
    x = np.array([1.0, 1.0, 1.0]) + rng.uniform(-1e-3, 1e-3, (P, 3))
    x[::97, 0] = 2e4
    p[::101, 1] = np.nan
    return p, x


def _run(lib, torch, p, x, layout, chunk, t_avg=None, capture=False, **kw):
    sw = lib.Sweep(model="lorenz", method="var", rtol=RTOL, atol=RTOL, h=1e-3, t_transient=2.0,
                   t_avg=6.0, dt_renorm=1.0, layout=layout, schedule="persistent", **kw)
    P = p.shape[0]
    spec, status, steps = np.empty((P, 3)), np.empty(P, np.int32), np.empty(P, np.int64)
    for o in range(0, P, chunk):
        def dev(a):
            a = a[o:o + chunk]
            return torch.from_numpy(np.ascontiguousarray(a.T if layout == "comp" and a.ndim == 2 else a)).cuda()
        dp, dx = dev(p), dev(x)
        n = min(chunk, P - o)
        ds = torch.zeros((n, 3) if layout == "point" else (3, n), dtype=torch.float64, device="cuda")
        st = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        sp = torch.zeros(n, dtype=torch.int64, device="cuda")
        ta = dev(t_avg) if t_avg is not None else None
        if capture:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                sw.run(dp, dx, ds, st, sp, t_avg=ta)
            g.replay()
        else:
            sw.run(dp, dx, ds, st, sp, t_avg=ta)
        torch.cuda.synchronize()
        a = ds.cpu().numpy()
        spec[o:o + n] = a.T if layout == "comp" else a
        status[o:o + n], steps[o:o + n] = st.cpu().numpy(), sp.cpu().numpy()
    sw.close()
    return spec, status, steps


@pytest.mark.parametrize("precision,integrator,layout", [
    ("fp64", "dverk65", "point"), ("fp64", "dopri5", "comp"), ("fp32", "dopri5", "comp"),
    ("fp32", "dverk65", "point")])
def test_two_launches_match_one(lib, precision, integrator, layout):
    import torch
    P = 120_001 if precision == "fp32" else 60_001  # above 1.5 waves, ragged
    p, x = _inputs(P)
    kw = dict(precision=precision, integrator=integrator)
    spec, status, steps = _run(lib, torch, p, x, layout, P, **kw)
    one, st1, sp1 = _run(lib, torch, p, x, layout, 20_000, **kw)
    assert np.array_equal(status, st1)
    assert (status[::97] != 0).all() and set(np.unique(status)) == {0, 1, 4}
    ok = status == 0
    assert np.isnan(spec[~ok]).all()
    assert np.array_equal(steps[~ok], sp1[~ok])
    d = np.abs(spec[ok] - one[ok])
    if precision == "fp64":
        # both are within the integration error, some 1e3 rtol over 8 units of
        # time at rates of 20
        assert d.max() < 1e3 * RTOL
    else:
        # FP32 renormalised at other times moves cells near a separatrix by up to
        # 1e-2: no further apart than two one-launch runs in other warps
        two, _, _ = _run(lib, torch, p, x, layout, 7001, **kw)
        own = np.abs(two[ok] - one[ok])
        assert np.sqrt((d ** 2).mean()) < 4 * np.sqrt((own ** 2).mean())
        assert d.max() < 4 * own.max()
    assert np.abs(steps[ok] - sp1[ok]).max() <= 0.1 * sp1[ok].max()


def test_two_launches_with_own_averaging_times_and_capture(lib):
    import torch
    P = 60_001
    p, x = _inputs(P, 8)
    t_avg = np.random.default_rng(1).uniform(1.0, 6.0, P)
    kw = dict(precision="fp64", integrator="dverk65")
    spec, status, _ = _run(lib, torch, p, x, "point", P, t_avg, **kw)
    one, st1, _ = _run(lib, torch, p, x, "point", 20_000, t_avg, **kw)
    ok = status == 0
    assert np.array_equal(status, st1)
    assert np.abs(spec[ok] - one[ok]).max() < 1e3 * RTOL
    # a captured sweep runs as one launch and owns no buffer of the handle's
    # beyond its point counter
    spec, status, _ = _run(lib, torch, p, x, "point", P, capture=True, **kw)
    one, st1, _ = _run(lib, torch, p, x, "point", 20_000, **kw)
    assert np.array_equal(status, st1)
    assert np.abs(spec[ok] - one[ok]).max() < 1e3 * RTOL


def test_sweeps_share_their_memory_across_handles_and_streams(lib):
    """Handles on streams of their own, made and closed while others run: each
    sweep has its own buffers until its last kernel is done."""
    import torch
    P = 60_001
    sets = [_inputs(P, seed) for seed in (11, 12, 13)]
    kw = dict(precision="fp64", integrator="dopri5")
    want = [_run(lib, torch, p, x, "point", 20_000, **kw) for p, x in sets]
    live, got = [], []
    for i in (0, 1, 2, 0, 1):
        p, x = (torch.from_numpy(a).cuda() for a in sets[i])
        ds = torch.zeros((P, 3), dtype=torch.float64, device="cuda")
        st = torch.full((P,), -1, dtype=torch.int32, device="cuda")
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        sw = lib.Sweep(model="lorenz", method="var", rtol=RTOL, atol=RTOL, h=1e-3,
                       t_transient=2.0, t_avg=6.0, dt_renorm=1.0, layout="point",
                       schedule="persistent", **kw)
        with torch.cuda.stream(s):
            sw.run(p, x, ds, st, None, stream=s.cuda_stream)
        live.append(sw)
        got.append((i, p, x, ds, st, s))
        if len(live) == 4:
            live.pop(0).close()
    torch.cuda.synchronize()
    for sw in live:
        sw.close()
    for i, _, _, ds, st, _ in got:
        spec, status, _ = want[i]
        ok = status == 0
        assert np.array_equal(st.cpu().numpy(), status)
        assert np.abs(ds.cpu().numpy()[ok] - spec[ok]).max() < 1e3 * RTOL
