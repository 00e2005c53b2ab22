"""The autotuner times the FP32 apply: the FP64 tiles, which the tile rule chose
for the FP64 kernels, stay as they were, and with them the bits of FP64 applies."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import femgpu  # noqa: E402


@pytest.mark.parametrize("n,p", [(48, 3), (80, 1), (12, 2)])
def test_autotune_leaves_fp64_tiles(n, p):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    op = femgpu.PADiffusionOperator((n, n, n), p)
    x = np.random.default_rng(n).standard_normal(op.n_dofs())
    before = {}
    for fmt in (femgpu.QDATA_AFFINE, femgpu.QDATA_FULL):
        op.set_qdata_format(fmt)
        before[fmt] = op.tile, op.matvec(x)
    (e,) = femgpu.batch_autotune([op], reps=2)
    assert e["us"][e["tz"]] == min(t for t in e["us"].values() if t is not None)
    for fmt, (tile, y) in before.items():
        op.set_qdata_format(fmt)
        assert op.tile == tile
        assert np.array_equal(op.matvec(x), y)
