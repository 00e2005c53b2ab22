"""A batched solve of an instance does not depend on the other members of the
batch: iterations, residual and solution have the same bits alone and beside
members that take most of the device."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import femgpu  # noqa: E402


def rhs(op, seed):
    b = np.random.default_rng(seed).standard_normal((op.NK, op.NJ, op.NI))
    b[[0, -1]], b[:, [0, -1]], b[:, :, [0, -1]] = 0.0, 0.0, 0.0
    return b.ravel()


@pytest.mark.parametrize("precond", [femgpu.PC_CHEBYSHEV, femgpu.PC_JACOBI])
def test_same_bits_in_every_batch(precond):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    # one piece, a few, many of either size; the large ones fill the device
    mine = [femgpu.PADiffusionOperator(s, p) for s, p in (((5, 6, 7), 1), ((11, 9, 10), 2), ((24, 23, 25), 2), ((30, 28, 33), 2))]
    big = [femgpu.PADiffusionOperator((40, 40, 40), 3) for _ in range(2)]
    cfg = femgpu.SolverConfig(rtol=1e-9, max_iter=2000, precision=femgpu.FP32_IR)
    seen = []
    for members in (mine, mine + big, big[:1] + mine[::-1], *([m] for m in mine)):
        xs = [np.zeros(m.n_dofs()) for m in members]
        ok, res = femgpu.batch_pcg(members, [rhs(m, m.n_dofs()) for m in members], xs, cfg, precond)
        assert ok
        seen.append({id(m): (r.iterations, r.true_residual, x.tobytes()) for m, r, x in zip(members, res, xs)})
    for m in mine:
        assert len({s[id(m)] for s in seen if id(m) in s}) == 1
