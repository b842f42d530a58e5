"""The surrogate's fused kernels (networks of width 64 and 128) at the edges of
their 64- and 128-row tiles, against the CPU FP64 backpropagation, and SiLU
where its fast division does not apply."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu

DOM = (5.0, 20.0, 0.0, 200.0)
# BF16 operands (unit roundoff 2^-9) through seven chained products: 7 x 2^-8
# in the worst case, relative to the whole gradient or output.
TOL = 7 * 2.0 ** -8


def _batch(n, seed=0):
    rng = np.random.default_rng(seed)
    xy = np.stack([rng.uniform(5, 20, n), rng.uniform(0, 200, n)], 1)
    return xy, rng.normal(size=(n, 3))


def _net(width, ensemble=2, seed=3):
    from chaos_oneapi_b200.surrogate import MLPEnsemble
    net = MLPEnsemble(ensemble=ensemble, width=width, outputs=3, seed=seed)
    net.set_domain(*DOM)
    return net


def _forward(p, width, xy):
    w = mo.unpack(p, width)
    h = mo.features(xy, DOM)
    for i in range(3):
        z = h @ w[2 * i] + w[2 * i + 1]
        h = np.where(z < -80.0, 0.0, mo.silu(np.maximum(z, -80.0)))
    return h @ w[6] + w[7]


@pytest.mark.parametrize("width", [64, 128])
@pytest.mark.parametrize("rows", [1, 63, 64, 65, 127, 129, 640])
def test_gradient_at_tile_edges(lib, width, rows):
    import torch
    net = _net(width)
    xy, T = _batch(rows)
    mean, std = np.zeros(3), np.ones(3)
    net.set_target_scale(mean, std)
    g, loss = net.gradient(torch.from_numpy(xy).cuda(), torch.from_numpy(T).cuda())
    params = net.get_params()
    for e in range(2):
        l_cpu, g_cpu = mo.loss_and_grad(params[e].astype(np.float64), width, xy, T, mean, std, DOM)
        rel = np.linalg.norm(g[e] - g_cpu) / np.linalg.norm(g_cpu)
        assert rel < TOL, (e, rel)
        assert abs(loss[e] - l_cpu) < TOL * max(1.0, l_cpu)
    net.close()


@pytest.mark.parametrize("width", [64, 128])
@pytest.mark.parametrize("rows", [1, 127, 128, 129, 5000])
def test_prediction_at_tile_edges(lib, width, rows):
    import torch
    net = _net(width, ensemble=3)
    net.set_target_scale([1.0, -2.0, 0.5], [0.5, 2.0, 1.0])
    xy, _ = _batch(rows, 5)
    mean, _ = net.predict(torch.from_numpy(xy).cuda())
    ys = np.stack([_forward(p.astype(np.float64), width, xy)[:, :3] for p in net.get_params()])
    want = (ys * [0.5, 2.0, 1.0] + [1.0, -2.0, 0.5]).mean(0)
    got = mean.cpu().numpy()
    assert np.linalg.norm(got - want) < TOL * np.linalg.norm(want)
    net.close()


def test_minibatch_rows_and_steps_match_the_gradient(lib):
    """One Adam step from zero moments moves every parameter by lr against the
    sign of its gradient; the minibatch is the whole (shuffled) set."""
    import torch
    net = _net(128)
    xy, T = _batch(200, 9)
    net.set_target_scale([0.0] * 3, [1.0] * 3)
    dxy, dT = torch.from_numpy(xy).cuda(), torch.from_numpy(T).cuda()
    g, _ = net.gradient(dxy, dT)
    before = net.get_params()
    net.train(dxy, dT, 1, 200, 1e-3, 0)
    step = net.get_params() - before
    big = np.abs(g) > 1e-4 * np.abs(g).max()
    np.testing.assert_allclose(step[big], -1e-3 * np.sign(g[big]), rtol=0, atol=1e-5)
    net.close()


def test_silu_where_the_exponential_overflows(lib):
    """Pre-activations of -100 (SiLU ~ -4e-42: zero in the next operand) and
    +100 in the same layer, against the FP64 forward pass."""
    import torch
    net = _net(128)
    net.set_target_scale([0.0] * 3, [1.0] * 3)
    p = net.get_params().copy()
    b1 = 16 * 128
    p[:, b1:b1 + 128:2] = -100.0
    p[:, b1 + 1:b1 + 128:8] = 100.0
    net.set_params(p)
    xy, T = _batch(130, 2)
    mean, _ = net.predict(torch.from_numpy(xy).cuda())
    want = np.stack([_forward(q.astype(np.float64), 128, xy)[:, :3] for q in p]).mean(0)
    assert np.linalg.norm(mean.cpu().numpy() - want) < TOL * np.linalg.norm(want)
    g, _ = net.gradient(torch.from_numpy(xy).cuda(), torch.from_numpy(T).cuda())
    assert np.isfinite(g).all()
    # a hidden unit held at -100 passes no gradient to its bias
    assert np.abs(g[:, b1:b1 + 128:2]).max() < 1e-30
    net.close()
