"""Lorenz-96's Gram-Schmidt at the edges of its 16-vector blocks, and sweeps in
two launches (all transients, then the averaging phases) against one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(lib, params, inits, k=40, **kw):
    cfg = dict(model="lorenz96", method="var", integrator="dopri5", precision="fp32", k=k,
               gs="mgs", rtol=1e-6, atol=1e-6, h=1e-2, max_steps=10_000_000)
    cfg.update(kw)
    with lib.Sweep(**cfg) as sw:
        return sw.run_host(np.ascontiguousarray(params), np.ascontiguousarray(inits),
                           want_steps=True)


@pytest.mark.parametrize("k", [1, 2, 15, 16, 17, 31, 32, 33, 39])
def test_partial_spectra_at_block_edges(lib, orc, k):
    """A settling cell's first k exponents against the FP64 oracle with the same
    k (the bound of the full spectrum's test)."""
    params = np.array([[3.0, 1.5], [2.0, 1.2]])
    inits = orc.make_inits(40, 2, [0.0] * 40, 0.01, 1, 3) + params[:, :1]
    kw = dict(t_transient=20.0, t_avg=20.0, dt_renorm=0.5)
    spec, st, _ = _run(lib, params, inits, k=k, **kw)
    want, wst, _ = orc.adaptive("lorenz96", params, inits, k, integrator="dopri5", gs="mgs",
                                rtol=1e-10, atol=1e-10, **kw)
    assert (st == 0).all() and (wst == 0).all()
    np.testing.assert_allclose(spec, want, rtol=0, atol=2e-3)


@pytest.mark.parametrize("layout", ["point", "comp"])
def test_two_launches_match_one_bit_for_bit(lib, layout):
    """More points than the GPU holds at once run in two launches, chunks of them
    in one; every point is a warp of its own, so nothing may change."""
    P, chunk = 5003, 1000
    rng = np.random.default_rng(6)
    p = np.stack([rng.uniform(4, 16, P), rng.uniform(0.5, 1.5, P)], 1)
    x = p[:, :1] + 0.01 * rng.standard_normal((P, 40))
    x[::61, 7] = 3e4      # outside the escape radius
    p[::67, 1] = np.nan
    t_avg = rng.uniform(0.2, 1.0, P)
    kw = dict(t_transient=0.5, t_avg=1.0, dt_renorm=0.5, layout=layout, k=13)

    def run(lo, hi):
        a = [v[lo:hi].T if layout == "comp" else v[lo:hi] for v in (p, x)]
        cfg = dict(model="lorenz96", method="var", integrator="dopri5", precision="fp32", gs="mgs",
                   rtol=1e-6, atol=1e-6, h=1e-2, **kw)
        with lib.Sweep(**cfg) as sw:
            spec, st, steps = sw.run_host(*[np.ascontiguousarray(v) for v in a],
                                          t_avg=t_avg[lo:hi].copy(), want_steps=True)
        return (spec.T if layout == "comp" else spec), st, steps

    whole = run(0, P)
    assert set(np.unique(whole[1])) == {0, 1, 4}
    for lo in range(0, P, chunk):
        hi = min(P, lo + chunk)
        for got, want in zip(run(lo, hi), whole):
            assert np.array_equal(got, want[lo:hi], equal_nan=True)
