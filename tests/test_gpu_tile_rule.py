"""Depths that the tile rule gives where counting whole rounds of CTAs is wrong:
the Q3 FP64 affine kernels, two CTAs on an SM of which share its FP64 pipe."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import femgpu  # noqa: E402


@pytest.mark.parametrize("n,depth", [
    (64, 7),  # nine items of 7 layers and one of 1; whole rounds gave one item of 16: 323 against 281 us
    (32, 2),
])
def test_q3_affine_depth(n, depth):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    op = femgpu.PADiffusionOperator((n, n, n), 3)
    op.set_qdata_format(femgpu.QDATA_AFFINE)
    assert op.tile[2] == depth
