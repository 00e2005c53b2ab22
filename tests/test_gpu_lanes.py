"""Both shapes of a warp's 32 elements (32 in x, and 8 in x by 4 in y) on the
same mesh: every apply form, the Jacobi diagonal and a re-tiled operator
against the oracle, at extents around the edges of the tiles (8 and 32 in x;
4, 8 and 16 rows in y; warps with no element), with the tolerances of the
other parity tests: 1e-12 relative in FP64, 2e-5 in FP32."""
import numpy as np
import pytest

from conftest import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import femgpu  # noqa: E402


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def native_f32(op, x, constrained):
    xn = torch.from_numpy(op.to_native(x).astype(np.float32)).cuda()
    yn = torch.zeros_like(xn)
    torch.cuda.synchronize()
    op.apply_native_f32(xn.data_ptr(), yn.data_ptr(), False, constrained)
    op.check()
    full = yn.cpu().numpy().astype(np.float64)
    assert np.all(full.reshape(op.NK, op.NJ, op.NIp)[:, :, op.NI:] == 0.0)
    return op.from_native(full)


@pytest.mark.parametrize("lanes", [8, 32])
@pytest.mark.parametrize("p,shape,tz", [
    (1, (9, 17, 5), 2), (1, (33, 4, 3), 1), (1, (7, 33, 9), 8),
    (2, (33, 18, 4), 2), (2, (8, 5, 3), 1), (2, (41, 3, 2), 4),
    (3, (9, 9, 3), 2), (3, (17, 5, 2), 1), (3, (1, 1, 1), 1),
])
def test_lane_shapes_match_oracle(lanes, p, shape, tz, monkeypatch):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    monkeypatch.setenv("FG_LANES_X", str(lanes))
    nx, ny, nz = shape
    rng = np.random.default_rng(nx + 10 * ny + p)
    E, q = nx * ny * nz, (p + 1) ** 3
    kq, rq = np.exp(rng.normal(size=E * q)), np.exp(0.3 * rng.normal(size=E * q))
    kind = (femgpu.DIFF, femgpu.MASS_DIFF, femgpu.MASS)[(nx + ny) % 3]
    mesh = O.Mesh(nx, ny, nz, p)
    coef = O.Coef(kind, c_m=0.7, c_k=1.3, kappa_q=kq, rho_q=rq)
    op = femgpu.PAOperator((nx, ny, nz), p, kind, kappa=kq, rho=rq, c_mass=0.7, c_diff=1.3, ess_tags=1 | 8 | 32)
    assert op.tile[0] == lanes
    mask = O.ess_mask(mesh, 1 | 8 | 32)
    x = rng.normal(size=op.n_dofs())
    raw, con = O.pa_apply(mesh, coef, x), O.apply_constrained(mesh, coef, mask, x)
    d = op.diagonal(constrained=True)
    for step in range(2):
        for fmt, tol in ((femgpu.QDATA_FULL, 1e-12), (femgpu.QDATA_AFFINE, 1e-12)):
            op.set_qdata_format(fmt)
            assert rel(op.matvec(x), raw) <= tol
            y = np.ones(op.n_dofs())
            op.apply(x, y, constrained=True)
            assert rel(y - 1.0, con) <= 1e-11  # the added ones cost up to four digits where y is small
            assert rel(native_f32(op, x, True), con) <= 2e-5
        op.set_qdata_format(femgpu.QDATA_FULL)
        assert rel(op.diagonal(constrained=True), d) <= 1e-13
        b = np.where(mask, 0.0, x)
        u = np.zeros(op.n_dofs())
        assert femgpu.solve_pcg_jacobi(op, b, u, femgpu.SolverConfig(rtol=1e-12, max_iter=5000)).converged
        assert rel(O.apply_constrained(mesh, coef, mask, u), b) <= 1e-10 or not np.any(b)
        op.set_tile(tz if step == 0 else 1)


def test_batch_of_both_lane_shapes(monkeypatch):
    """One batch whose members take different lane shapes: the same
    iterations as their single solves within 2, solutions to 1e-7."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    shapes = [(32, 6, 5), (9, 16, 8), (33, 33, 6)]
    ops = []
    for s, lanes in zip(shapes, (32, 8, 8)):
        monkeypatch.setenv("FG_LANES_X", str(lanes))
        ops.append(femgpu.PADiffusionOperator(s, 2))
    assert {o.tile[0] for o in ops} == {8, 32}
    rng = np.random.default_rng(4)
    bs = []
    for o, s in zip(ops, shapes):
        b = rng.normal(size=o.n_dofs())
        b[O.ess_mask(O.Mesh(*s, 2), 63) == 1] = 0.0
        bs.append(b)
    cfg = femgpu.SolverConfig(rtol=1e-10, precision=femgpu.FP32_IR)
    xs = [np.zeros_like(b) for b in bs]
    ok, res = femgpu.batch_pcg(ops, bs, xs, cfg)
    assert ok
    for o, b, x, r in zip(ops, bs, xs, res):
        one = np.zeros_like(b)
        single = femgpu.solve_pcg_chebyshev(o, b, one, cfg)
        assert single.converged and abs(single.iterations - r.iterations) <= 2
        assert rel(x, one) <= 1e-7
