"""What the first FP32 call of a handle builds: an affine handle's takes no
full-format FP32 copy of the quadrature data (it would not read it), whichever
way the handle came to its format; both formats stay usable after a switch."""
import numpy as np
import pytest

from conftest import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import femgpu  # noqa: E402


def apply(op, x):
    xn = torch.from_numpy(op.to_native(x).astype(np.float32)).cuda()
    yn = torch.zeros_like(xn)
    torch.cuda.synchronize()
    op.apply_native_f32(xn.data_ptr(), yn.data_ptr(), False, False)
    op.check()
    return op.from_native(yn.cpu().numpy().astype(np.float64))


def test_affine_handle_builds_no_full_copy():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n, p = 40, 3
    op = femgpu.PADiffusionOperator((n, n, n), p)
    op.set_qdata_format(femgpu.QDATA_AFFINE)
    x = np.random.default_rng(0).standard_normal(op.n_dofs())
    native = torch.from_numpy(op.to_native(x).astype(np.float32)).cuda()
    out = torch.zeros_like(native)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    op.apply_native_f32(native.data_ptr(), out.data_ptr(), False, False)
    op.check()
    grown = free - torch.cuda.mem_get_info()[0]
    points = 64 * 4 * n ** 3  # bytes of one FP32 value per point
    # the affine data (one value a point and six an element), eleven vectors, the
    # face slots and the allocator's rounding; the full format would add six values a point
    assert grown < 2 * points + 11 * native.numel() * 4 + (32 << 20)


@pytest.mark.parametrize("p,shape", [(1, (33, 6, 5)), (2, (9, 17, 5)), (3, (5, 6, 7))])
def test_formats_alternate(p, shape):
    """Full and affine FP32 applies in turn, either first, within 2e-5 of the oracle."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    for first in (femgpu.QDATA_AFFINE, femgpu.QDATA_FULL):
        op = femgpu.PADiffusionOperator(shape, p)
        x = np.random.default_rng(p).standard_normal(op.n_dofs())
        ref = O.pa_apply(O.Mesh(*shape, p), O.Coef(O.DIFF), x)
        for fmt in (first, 1 - first, first):
            op.set_qdata_format(fmt)
            assert np.linalg.norm(apply(op, x) - ref) <= 2e-5 * np.linalg.norm(ref)
        op.set_tile(2)
        assert np.linalg.norm(apply(op, x) - ref) <= 2e-5 * np.linalg.norm(ref)
