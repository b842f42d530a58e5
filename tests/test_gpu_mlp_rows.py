"""The fused training and prediction kernels beyond one round of their buffers:
more than five 128-row tiles (the weight gradients' stages are reused), more
than eight (the bias gradients'), rows past a chunk of a prediction, and a
smaller call after a larger one."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu

DOM = (5.0, 20.0, 0.0, 200.0)
TOL = 7 * 2.0 ** -8  # BF16 operands through seven chained products


def _inputs(rows, seed=0):
    rng = np.random.default_rng(seed)
    xy = np.stack([rng.uniform(5, 20, rows), rng.uniform(0, 200, rows)], 1)
    return xy, rng.normal(size=(rows, 3))


def _net(width, ensemble=2):
    from chaos_oneapi_b200.surrogate import MLPEnsemble
    net = MLPEnsemble(ensemble=ensemble, width=width, outputs=3, seed=3)
    net.set_domain(*DOM)
    net.set_target_scale([0.0] * 3, [1.0] * 3)
    return net


def _cuda(*arrays):
    import torch
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


@pytest.mark.parametrize("width", [64, 128])
@pytest.mark.parametrize("rows", [641, 768, 1024, 1025, 1153, 2500])
@pytest.mark.parametrize("heavy", ["none", "last", "middle"])
def test_gradient_of_many_tiles(lib, width, rows, heavy):
    """heavy: one row's target is so far off that the gradient is nearly its own,
    so that losing or doubling that row alone shows."""
    net = _net(width)
    xy, T = _inputs(rows)
    if heavy != "none":
        T[rows - 1 if heavy == "last" else rows // 2] = 1000.0
    g, loss = net.gradient(*_cuda(xy, T))
    params = net.get_params()
    for e in range(2):
        l_cpu, g_cpu = mo.loss_and_grad(params[e].astype(np.float64), width, xy, T, np.zeros(3),
                                        np.ones(3), DOM)
        assert np.linalg.norm(g[e] - g_cpu) < TOL * np.linalg.norm(g_cpu)
        # the biases alone: their sums are kernels of their own
        for got, want in zip(mo.unpack(g[e], width)[1::2], mo.unpack(g_cpu, width)[1::2]):
            if heavy != "none":
                assert np.linalg.norm(got - want) < TOL * np.linalg.norm(want)
        assert abs(loss[e] - l_cpu) < TOL * max(1.0, l_cpu)
    net.close()


@pytest.mark.parametrize("width", [64, 128])
def test_smaller_call_after_a_larger_one(lib, width):
    big, small = _cuda(*_inputs(2500)), _cuda(*_inputs(130, 4))
    used, fresh = _net(width), _net(width)
    used.gradient(*big)
    used.predict(big[0])
    assert np.array_equal(used.gradient(*small)[0], fresh.gradient(*small)[0])
    for a, b in zip(used.predict(small[0]), fresh.predict(small[0])):
        assert np.array_equal(a.cpu().numpy(), b.cpu().numpy())
    used.close()
    fresh.close()


@pytest.mark.parametrize("width", [64, 128])
@pytest.mark.parametrize("rows", [30_011, (1 << 18) + 129])
def test_predicted_rows_do_not_depend_on_their_tile(lib, width, rows):
    """Every row of a prediction of many tiles (and of two chunks) has the bits
    of a prediction of 4,000 rows, which starts every group's tiles afresh."""
    net = _net(width, ensemble=3)
    xy, _ = _cuda(*_inputs(rows, 7))
    mean, std = (a.cpu().numpy() for a in net.predict(xy))
    for lo in range(0, rows, 4000):
        m, s = net.predict(xy[lo:lo + 4000].contiguous())
        assert np.array_equal(m.cpu().numpy(), mean[lo:lo + 4000])
        assert np.array_equal(s.cpu().numpy(), std[lo:lo + 4000])
    net.close()
