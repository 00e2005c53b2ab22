"""The Q3 FP64 unstructured apply has two plans of its shared memory, chosen by the
rounds of CTAs: meshes of either (one round; 343 chunks of up to 2,450 DOFs, two rounds of
two CTAs per SM or one of three), every kind, against the structured operator of the
same box (1e-12)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import bench  # noqa: E402
import femgpu  # noqa: E402


@pytest.mark.parametrize("n", [8, 11, 28])
@pytest.mark.parametrize("kind", [femgpu.MASS, femgpu.DIFF, femgpu.MASS_DIFF])
@pytest.mark.parametrize("constrained", [False, True])
def test_q3_plans_match_box(n, kind, constrained):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    coords, conn, maps = bench.box_as_hex_mesh(n, 3)
    sn = 3 * n + 1
    ids = np.arange(sn ** 3).reshape(sn, sn, sn)
    ess = np.unique(np.concatenate([ids[[0, -1]].ravel(), ids[:, [0, -1]].ravel(), ids[:, :, [0, -1]].ravel()]))
    hexop = femgpu.HexMeshOperator(3, coords, conn, elem_dofs=maps, n_dofs=sn ** 3, kind=kind,
                                   ess_dofs=ess.astype(np.uint32))
    box = femgpu.PAOperator((n, n, n), 3, kind)
    x = np.random.default_rng(n).standard_normal(sn ** 3)
    want = box.matvec(x, constrained=constrained)
    for _ in range(2):
        y = hexop.matvec(x, constrained=constrained)
        assert np.linalg.norm(y - want) <= 1e-12 * np.linalg.norm(want)
