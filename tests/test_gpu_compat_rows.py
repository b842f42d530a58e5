"""The fixed-step sweep's two launch forms -- one lane per row of a point (few
points) and one thread per point -- bit for bit against each other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = {
    "shimizu": ([0.8, 0.5], [0.1, 0.05, 0.02]),
    "lorenz": ([10.0, 28.0, 8.0 / 3.0], [1.0, 1.0, 1.0]),
    "rossler": ([0.2, 0.2, 5.7], [1.0, 1.0, 0.0]),
    "chua": ([9.0, 14.3, -8.0 / 7.0, -5.0 / 7.0], [0.1, 0.0, 0.0]),
    "hyper_rossler": ([0.5, 0.05], [-10.0, -6.0, 0.0, 10.0]),
}


@pytest.mark.parametrize("model", list(CASES))
@pytest.mark.parametrize("method", ["fd", "var", "qr"])
@pytest.mark.parametrize("k", [1, 2, 3, 4])
def test_rows_match_threads(lib, model, method, k):
    import torch
    pb, xb = CASES[model]
    n = len(xb)
    if k > n or (method == "qr" and k != n):
        pytest.skip("k <= dimension; QR takes all columns")
    P = 20_011  # above the rows form's range on any B200; ragged
    rng = np.random.default_rng(4)
    p = np.array(pb) * (1 + 0.05 * rng.uniform(-1, 1, (P, len(pb))))
    x = np.array(xb) + rng.uniform(-1e-3, 1e-3, (P, n))
    p[5, 0] = np.nan
    add = 0.05 / 0.01

    def run(lo, hi, accumulate):
        d = [torch.from_numpy(a[lo:hi].copy()).cuda() for a in (p, x)]
        out = torch.full((hi - lo, k), accumulate, dtype=torch.float64, device="cuda")
        close = torch.zeros((hi - lo, k * n), dtype=torch.float64, device="cuda")
        lib.cuda_lyapunov(hi - lo, method == "qr", method == "var", d[1],
                          close, n, model, d[0], len(pb), 1e-7, 0.01, out, k, 0.2, 0.1, 0.35, add)
        torch.cuda.synchronize()
        return [t.cpu().numpy() for t in (out, d[1], close)]

    whole = run(0, P, 0.25)
    for lo, hi in ((0, 1), (1, 8), (8, 1003), (1003, 12_003)):
        for got, want in zip(run(lo, hi, 0.25), whole):
            assert np.array_equal(got, want[lo:hi], equal_nan=True), (lo, hi)


@pytest.mark.parametrize("t_calc", [0.005, 0.01, 0.02])
def test_rows_of_few_steps(lib, t_calc):
    """One and two steps (QR's state runs a step ahead), component-major."""
    import torch
    P = 15_000
    p, x = CASES["lorenz"]
    rng = np.random.default_rng(2)
    p = np.array(p) + rng.uniform(-1, 1, (P, 3))
    x = np.array(x) + rng.uniform(-1, 1, (P, 3))
    for method in ("qr", "var", "fd"):
        sw = lib.Sweep(model="lorenz", method=method, integrator="dverk", precision="compat", k=3,
                       eps=1e-7, h=0.01, t_transient=0.0, t_align=0.0, t_avg=t_calc,
                       dt_renorm=0.01, layout="comp")

        def run(lo, hi):
            d = [torch.from_numpy(np.ascontiguousarray(a[lo:hi].T)).cuda() for a in (p, x)]
            out = torch.zeros((3, hi - lo), dtype=torch.float64, device="cuda")
            st = torch.full((hi - lo,), -1, dtype=torch.int32, device="cuda")
            sw.run(d[0], d[1], out, st)
            sw.sync()
            return out.cpu().numpy(), d[1].cpu().numpy(), st.cpu().numpy()[None]
        whole, part = run(0, P), run(77, 1000)
        for got, want in zip(part, whole):
            assert np.array_equal(got, want[:, 77:1000])
        sw.close()
