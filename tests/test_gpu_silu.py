"""SiLU of the fused networks (widths 64 and 128): its division by Newton's
method and its chunked form against the plain functions on every 32-bit float,
and a pre-activation of +infinity through a whole prediction."""
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def counts(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path_factory.mktemp("silu") / "silu_driver")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "-I" + os.path.join(os.path.dirname(HERE), "include"), "-o", exe,
                    os.path.join(HERE, "device", "silu_driver.cu")], check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return {f[0]: tuple(int(v) for v in f[1:]) for f in map(str.split, out.splitlines())}


@pytest.mark.parametrize("name", ["silu", "silu_alone", "dsilu", "quotient", "reciprocal"])
def test_every_float(counts, name):
    """The quotient is the correctly rounded one, so nothing differs."""
    seen, differ, ulps = counts[name]
    assert seen > 1 << 29
    assert (differ, ulps) == (0, 0)


@pytest.mark.parametrize("width", [64, 128])
def test_infinite_preactivation(lib, width):
    """SiLU(+inf) = +inf: with positive weights the infinity reaches the output;
    SiLU(-inf) = -inf / inf is NaN."""
    import torch
    from chaos_oneapi_b200.surrogate import MLPEnsemble
    net = MLPEnsemble(ensemble=1, width=width, outputs=3, seed=0)
    net.set_domain(5.0, 20.0, 0.0, 200.0)
    net.set_target_scale([0.0] * 3, [1.0] * 3)
    rng = np.random.default_rng(0)
    xy = torch.from_numpy(np.stack([rng.uniform(5, 20, 130), rng.uniform(0, 200, 130)], 1)).cuda()
    p = np.full_like(net.get_params(), 1.0 / 64)
    b1 = 16 * width
    for value, units in ((np.inf, slice(b1, b1 + width)), (np.inf, slice(b1 + 3, b1 + 4))):
        q = p.copy()
        q[:, units] = value
        net.set_params(q)
        mean, _ = net.predict(xy)
        assert (mean.cpu().numpy() == np.inf).all()
    q = p.copy()
    q[:, b1 + 3] = -np.inf
    net.set_params(q)
    mean, _ = net.predict(xy)
    assert np.isnan(mean.cpu().numpy()).all()
    net.close()
