"""The sums of the weight and bias gradients over a large volume.  With zero
weights and a bias of one in front of the last convolution its gradients are
sums of the rounded output gradient alone, all of one sign, and are known in
64 bits.  A partial sum covers at most 4,096 voxels, 256 steps of the tensor core;
the partials are added in FP32.  An addition is off by at most 2^-24 of the sum, half
of that on average over a growing sum, and m of them by sqrt(m) as much: three
times (sqrt(256) + sqrt(partials)) 2^-25."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import femgpu  # noqa: E402
import unet_ref as R  # noqa: E402  (oracle/unet_ref.py)

from conftest import oracle as O  # noqa: E402,F401  (path of the oracle)


@pytest.mark.parametrize("shape", [(1, 129, 129, 129), (3, 33, 65, 41)])
def test_last_layer_sums(shape):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    net = femgpu.UNet(seed=0)
    params = np.zeros(net.num_params, dtype=np.float32)
    at, o = {}, 0
    for name, (ci, co) in zip(R.LAYERS, R.layer_shapes()):
        at[name] = o, o + co * 27 * ci, o + co * 27 * ci + co
        o = at[name][2]
    params[at["l0c"][1]:at["l0c"][2]] = 1.0
    net.set_params(params)
    rng = np.random.default_rng(2)
    tgt = rng.uniform(0.5, 1.5, size=shape).astype(np.float32)
    net.loss_grad(rng.standard_normal(shape + (2,)).astype(np.float32), tgt)
    g = net.get_grads().astype(np.float64)
    d = R.bf16(-2.0 * tgt.astype(np.float64) / tgt.size)
    n = tgt.size
    bound = 3 * (16 + np.sqrt(n / 4096)) * 2.0 ** -25
    b = g[at["out"][1]]
    assert abs(b - d.sum()) <= bound * abs(d.sum())
    w = g[at["out"][0]:at["out"][1]].reshape(-1, 27, 16)[0]
    for tap in range(27):
        sl = tuple(slice(max(0, -k), shape[a + 1] - max(0, k))
                   for a, k in enumerate((tap // 9 - 1, tap // 3 % 3 - 1, tap % 3 - 1)))
        exact = d[(slice(None),) + sl].sum()
        assert np.all(np.abs(w[tap] - exact) <= bound * abs(exact))
