"""Two networks trained at the same time on streams of their own: their kernels
share the SMs and the tensor memory, and a step's kernels start before the
previous ones have ended, yet each network ends with the bits it has alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _net(width, seed):
    from chaos_oneapi_b200.surrogate import MLPEnsemble
    net = MLPEnsemble(ensemble=4, width=width, outputs=3, seed=seed)
    net.set_domain(5.0, 20.0, 0.0, 200.0)
    net.set_target_scale([0.0] * 3, [1.0] * 3)
    return net


@pytest.mark.parametrize("widths", [(64, 64), (64, 128), (128, 128)])
def test_concurrent_training(lib, widths):
    import torch
    rng = np.random.default_rng(1)
    xy = torch.from_numpy(np.stack([rng.uniform(5, 20, 4096), rng.uniform(0, 200, 4096)], 1)).cuda()
    T = torch.from_numpy(rng.normal(size=(4096, 3))).cuda()
    torch.cuda.synchronize()
    steps = 200

    def train(net, stream):
        net.train(xy, T, steps, 1000, 1e-3, 5, stream=stream.cuda_stream)

    want = []
    for i, w in enumerate(widths):
        net = _net(w, i)
        train(net, torch.cuda.Stream())
        want.append(net.get_params())
        net.close()
    nets = [_net(w, i) for i, w in enumerate(widths)]
    streams = [torch.cuda.Stream() for _ in nets]
    threads = [threading.Thread(target=train, args=a) for a in zip(nets, streams)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for net, w in zip(nets, want):
        assert np.array_equal(net.get_params(), w)
        net.close()
