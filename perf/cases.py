"""Workloads of the operator library, for timing and for comparing outputs.

Each case goes through the package's public entry points the way a solver
program does: the operator is built once, vectors stay where such a program
keeps them, and one pass is one apply, one solve or one training step.

Families
  box    one constrained apply on a structured hexahedral box, device vectors in
         the native layout (what a Krylov or time-stepping loop calls)
  hex    the same on an unstructured Hex8 mesh with the caller's element maps
  tet    the same on an unstructured tetrahedral mesh (TetP1 to TetP3)
  pcg    one whole preconditioned solve
  batch  many uneven solves together
  unet   one training step's loss and gradients of the learned correction

Sizes are those of the benchmark (128^3 Q2 apply, 64^3 Q2 heat stage, batches
of 8^3 to 48^3 elements of orders 1 to 3, the 24^3 Q1 Poisson example, the
33^3 network volume) and odd ones of the same ranges.
"""
import functools
import itertools
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fem-rs_b200"))

import femgpu  # noqa: E402
from femgpu import tet as tetmesh  # noqa: E402
from femgpu.fields import lognormal_kappa_q  # noqa: E402

MASS, DIFF, MASS_DIFF = femgpu.MASS, femgpu.DIFF, femgpu.MASS_DIFF


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # The smallest member of a batch of unrelated problems, applied on its own: launch latency.
        _box("box_q2_8", 8, 8, 8, 2),
        # The benchmark's operator: one FP64 apply of a 17M-DOF Poisson problem with lognormal coefficient.
        _box("box_q2_128", 128, 128, 128, 2),
        # A curved (perturbed) Q3 mesh whose extents fit no tile: the drop-in FP64 apply of a user's own box.
        _box("box_q3_ragged", 45, 41, 38, 3, geometry="perturbed"),
        # The smoother's apply of a mixed-precision solve of a Q3 box as it occurs in batches.
        _box("box_q3_f32_affine", 48, 48, 48, 3, bits=32, fmt="affine"),
        # The stage operator M + gamma dt K of the heat example in its fastest form.
        _box("box_q2_f32_stage", 64, 64, 64, 2, kind=MASS_DIFF, bits=32, fmt="affine"),
        # A mesh generator's hexahedra with the DOF numbering of its own DofManager.
        _hex("hex_q2_64", 64, 64, 64, 2),
        # Tetrahedral Poisson, quadratic elements, coefficient at the quadrature points.
        _tet("tet_p2", 40, 2),
        # The reaction-diffusion operator on cubic tetrahedra (mass term: the points of a degree-7 rule).
        _tet("tet_p3_mass_diff", 20, 3, kind=MASS_DIFF),
        # The drop-in call of the Poisson example: Jacobi-PCG on host arrays, 15,625 DOFs.
        _pcg("pcg_jacobi_24", 24, 24, 24, 1, "jacobi", 64, "host", "perturbed"),
        # The solver's recommended form: Chebyshev(4)-preconditioned, FP32 inside FP64 residuals.
        _pcg("pcg_mixed_cheb", 48, 40, 44, 2, "chebyshev", 32, "device", "uniform"),
        # Uneven independent problems solved together (parameter studies, subdomains).
        dict(name="batch_16", family="batch", count=16, lo=8, hi=48, sizes=3),
        # One training step's loss and gradients on the network volume of the 128^3 Q2 solve.
        dict(name="unet_33", family="unet", batch=1, nz=33, ny=33, nx=33),
    ]


def _box(name, nx, ny, nz, p, kind=DIFF, bits=64, fmt="full", geometry="uniform"):
    return dict(name=name, family="box", nx=nx, ny=ny, nz=nz, p=p, kind=kind, bits=bits, fmt=fmt, geometry=geometry)


def _hex(name, nx, ny, nz, p, kind=DIFF, bits=64):
    return dict(name=name, family="hex", nx=nx, ny=ny, nz=nz, p=p, kind=kind, bits=bits)


def _tet(name, n, p, kind=DIFF):
    return dict(name=name, family="tet", n=n, p=p, kind=kind)


def _pcg(name, nx, ny, nz, p, precond, bits, memory, geometry):
    return dict(name=name, family="pcg", nx=nx, ny=ny, nz=nz, p=p, precond=precond, bits=bits, memory=memory,
                geometry=geometry)


def _extent(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above; applies most often, as they are called most often."""
    family = rng.choice(["box"] * 6 + ["hex"] * 2 + ["tet"] * 2 + ["pcg"] * 2 + ["batch", "unet"])
    if family == "box":
        p = rng.choice([1, 2, 3])
        top = {1: 192, 2: 112, 3: 64}[p]
        c = _box(None, _extent(rng, 6, top), _extent(rng, 6, top), _extent(rng, 6, top), p,
                 kind=rng.choice([DIFF, DIFF, MASS_DIFF, MASS]), bits=rng.choice([64, 64, 32]),
                 fmt=rng.choice(["full", "full", "affine"]), geometry=rng.choice(["uniform", "perturbed"]))
        if c["fmt"] == "affine":  # elements with a constant Jacobian only
            c["geometry"] = "uniform"
    elif family == "hex":
        p = rng.choice([1, 2, 3])
        top = {1: 80, 2: 64, 3: 36}[p]
        c = _hex(None, _extent(rng, 6, top), _extent(rng, 6, top), _extent(rng, 6, top), p,
                 kind=rng.choice([DIFF, DIFF, MASS_DIFF, MASS]), bits=rng.choice([64, 64, 32]))
    elif family == "tet":
        p = rng.choice([1, 2, 3])
        c = _tet(None, _extent(rng, 5, {1: 56, 2: 40, 3: 22}[p]), p, kind=rng.choice([DIFF, DIFF, MASS_DIFF, MASS]))
    elif family == "pcg":
        p = rng.choice([1, 2, 3])
        top = {1: 64, 2: 40, 3: 24}[p]
        c = _pcg(None, _extent(rng, 8, top), _extent(rng, 8, top), _extent(rng, 8, top), p,
                 rng.choice(["jacobi", "chebyshev", "none"]), 64, rng.choice(["host", "device"]),
                 rng.choice(["uniform", "perturbed"]))
        if c["precond"] != "none" and rng.random() < 0.5:
            c["bits"] = 32
    elif family == "batch":
        lo = rng.randint(6, 16)
        c = dict(family="batch", count=rng.randint(2, 12), lo=lo, hi=lo + rng.randint(4, 32), sizes=rng.randint(0, 10 ** 6))
    else:
        c = dict(family="unet", batch=rng.randint(1, 2), nz=4 * rng.randint(1, 8) + 1, ny=4 * rng.randint(1, 8) + 1,
                 nx=4 * rng.randint(1, 8) + 1)
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------
# reference elements in 64 bits (torch / numpy, nothing of the package)
# ---------------------------------------------------------------------------
def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return x, w


def _lagrange(p, x):
    """(values, derivatives) [q, d] of the equispaced Lagrange polynomials on [-1, 1]."""
    nodes = np.linspace(-1.0, 1.0, p + 1)
    B, G = np.zeros((len(x), p + 1)), np.zeros((len(x), p + 1))
    for d in range(p + 1):
        c = np.poly1d(1.0)
        for k in range(p + 1):
            if k != d:
                c = c * np.poly1d([1.0, -nodes[k]]) / (nodes[d] - nodes[k])
        B[:, d], G[:, d] = c(x), c.deriv()(x)
    return B, G


@functools.lru_cache(None)
def _hex_element(p):
    """Basis [q, l], gradients [q, l, 3], weights [q], trilinear vertex gradients [q, 8, 3]; point and local DOF
    order (z, y, x), x fastest; vertices in the same order."""
    x, w = _gauss(p + 1)
    out = []
    for order in (p, 1):
        B, G = _lagrange(order, x)
        phi = np.einsum("zc,yb,xa->zyxcba", B, B, B)
        g = np.stack([np.einsum("zc,yb,xa->zyxcba", B, B, G), np.einsum("zc,yb,xa->zyxcba", B, G, B),
                      np.einsum("zc,yb,xa->zyxcba", G, B, B)], axis=-1)
        q, n = (p + 1) ** 3, (order + 1) ** 3
        out += [phi.reshape(q, n), g.reshape(q, n, 3)]
    return out[0], out[1], np.einsum("z,y,x->zyx", w, w, w).ravel(), out[3]


def _grundmann_moeller(s):
    """Points [q, 3] and weights of the Grundmann-Moeller rule of degree 2s + 1 on the unit tetrahedron."""
    pts, wts = [], []
    for i in range(s + 1):
        m, d = s - i, 2 * s + 1
        w = (-1) ** i * 2.0 ** (-2 * s) * (d + 3 - 2 * i) ** d / (math.factorial(i) * math.factorial(d + 3 - i))
        for b in itertools.product(range(m + 1), repeat=4):
            if sum(b) == m:
                pts.append([(2 * b[k] + 1) / (d + 3 - 2 * i) for k in (1, 2, 3)])
                wts.append(w)
    return np.array(pts), np.array(wts)


@functools.lru_cache(None)
def _tet_element(p, kind):
    """Quadrature order, points [q, 3], basis [q, l], gradients [q, l, 3], weights [q] of TetP1 to TetP3."""
    order = 2 * p + (1 if kind & MASS else 0)
    if order <= 2:
        a, b = 0.1381966011250105, 0.5854101966249685
        xi, w = np.array([[a, a, a], [b, a, a], [a, b, a], [a, a, b]]), np.full(4, 1 / 24)
    else:
        xi, w = _grundmann_moeller(2 if order <= 5 else 3)
    # the Lagrange basis of the nodes, from the monomials of degree <= p
    vert = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]], dtype=float)
    edges = [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]
    nodes = [v for v in vert]
    for i, j in edges:
        nodes += [((p - k) * vert[i] + k * vert[j]) / p for k in range(1, p)]
    if p == 3:
        nodes += [(vert[i] + vert[j] + vert[k]) / 3 for i, j, k in ((0, 1, 2), (0, 1, 3), (0, 2, 3), (1, 2, 3))]
    nodes = np.array(nodes)
    ex = [e for e in itertools.product(range(p + 1), repeat=3) if sum(e) <= p]

    def mono(x, dif=None):
        cols = []
        for e in ex:
            c = np.ones(len(x))
            for a in range(3):
                k = e[a]
                if dif == a:
                    c = c * (k * x[:, a] ** (k - 1) if k else 0.0)
                else:
                    c = c * x[:, a] ** k
            cols.append(c)
        return np.stack(cols, axis=1)

    C = np.linalg.inv(mono(nodes))
    return order, xi, mono(xi) @ C, np.stack([mono(xi, a) @ C for a in range(3)], axis=-1), w


class _Plain:
    """y = A x in 64 bits, element by element: gather, dense element products, scatter; identity on the
    essential DOFs."""

    def __init__(self, dofs, n, phi, grad, w, vgrad, xyz, kind, kappa, rho, c_mass, c_diff, ess):
        dev = "cuda"
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
        self.dofs, self.n = torch.as_tensor(dofs, dtype=torch.int64, device=dev), n
        self.phi, self.grad, self.kind = t(phi), t(grad), kind
        self.ess = torch.as_tensor(ess, dtype=torch.bool, device=dev)
        E, q = self.dofs.shape[0], len(w)
        self.D = torch.empty((E, q, 3, 3), dtype=torch.float64, device=dev) if kind & DIFF else None
        self.m = torch.empty((E, q), dtype=torch.float64, device=dev) if kind & MASS else None
        xyz, vg, w = t(xyz), t(vgrad), t(w)
        for s in self._parts():
            J = torch.einsum("evi,qvd->eqid", xyz[s], vg)
            det = torch.linalg.det(J).abs() * w
            if kind & DIFF:
                inv = torch.linalg.inv(J)
                self.D[s] = c_diff * (det * self._at(kappa, s))[..., None, None] * (inv @ inv.transpose(-1, -2))
            if kind & MASS:
                self.m[s] = c_mass * det * self._at(rho, s)

    def _parts(self):
        return [slice(a, a + (1 << 18)) for a in range(0, self.dofs.shape[0], 1 << 18)]

    @staticmethod
    def _at(c, s):
        return c if isinstance(c, float) else torch.as_tensor(c[s], dtype=torch.float64, device="cuda")

    def __call__(self, x):
        y = torch.zeros(self.n, dtype=torch.float64, device="cuda")
        xm = x.masked_fill(self.ess, 0.0)
        for s in self._parts():
            u = xm[self.dofs[s]]
            r = torch.zeros_like(u)
            if self.kind & DIFF:
                g = torch.einsum("el,qld->eqd", u, self.grad)
                r += torch.einsum("eqd,qld->el", torch.einsum("eqcd,eqd->eqc", self.D[s], g), self.grad)
            if self.kind & MASS:
                r += (self.m[s] * (u @ self.phi.T)) @ self.phi
            y.index_add_(0, self.dofs[s].reshape(-1), r.reshape(-1))
        return torch.where(self.ess, x, y)

    def diagonal(self):
        d = torch.zeros(self.n, dtype=torch.float64, device="cuda")
        for s in self._parts():
            r = torch.zeros(self.dofs[s].shape, dtype=torch.float64, device="cuda")
            if self.kind & DIFF:
                for a in range(3):
                    for b in range(3):
                        r += self.D[s][..., a, b] @ (self.grad[..., a] * self.grad[..., b])
            if self.kind & MASS:
                r += self.m[s] @ (self.phi ** 2)
            d.index_add_(0, self.dofs[s].reshape(-1), r.reshape(-1))
        return d.masked_fill(self.ess, 1.0)

    def solve(self, b, rtol=1e-14, most=20000):
        """Jacobi-preconditioned CG to the limit of 64 bits."""
        inv = 1.0 / self.diagonal()
        x, r = torch.zeros_like(b), b.clone()
        z = inv * r
        p, rz, nb = z.clone(), torch.dot(r, z), b.norm()
        for k in range(most):
            ap = self(p)
            a = rz / torch.dot(p, ap)
            x += a * p
            r -= a * ap
            if k % 20 == 0 and r.norm() <= rtol * nb:
                break
            z = inv * r
            new = torch.dot(r, z)
            p = z + (new / rz) * p
            rz = new
        return x


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _grid(nx, ny, nz, p):
    return nx * p + 1, ny * p + 1, nz * p + 1


@functools.lru_cache(8)
def _box_maps(nx, ny, nz, p):
    """Element DOF map [E, (p+1)^3] and vertex map [E, 8], both (z, y, x) with x fastest; boundary mask."""
    def maps(order):
        NI, NJ, NK = _grid(nx, ny, nz, order)
        k, j, i = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
        base = ((k * NJ + j) * NI + i).reshape(-1, 1) * order
        o = np.arange(order + 1)
        off = ((o[:, None, None] * NJ + o[None, :, None]) * NI + o[None, None, :]).reshape(1, -1)
        return base + off
    NI, NJ, NK = _grid(nx, ny, nz, p)
    ess = np.zeros((NK, NJ, NI), dtype=bool)
    ess[[0, -1]] = True
    ess[:, [0, -1]] = True
    ess[:, :, [0, -1]] = True
    return maps(p), maps(1), ess.ravel()


def _vertices(case, rng, amount=0.2):
    """Vertices of the unit cube's grid; interior ones moved by up to `amount` of a cell."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    v = femgpu.unit_cube_vertices(nx, ny, nz)
    inner = np.all((v > 1e-12) & (v < 1 - 1e-12), axis=1)
    v[inner] += amount * rng.uniform(-1, 1, size=(int(inner.sum()), 3)) / np.array([nx, ny, nz])
    return v


def _box_inputs(case, seed):
    """(vertices or None, kappa, rho) of a structured case."""
    nx, ny, nz, p = case["nx"], case["ny"], case["nz"], case["p"]
    vc = _vertices(case, np.random.default_rng(seed)) if case.get("geometry") == "perturbed" else None
    kappa = lognormal_kappa_q(nx, ny, nz, p, seed=seed, device="cuda") if case.get("kind", DIFF) & DIFF else 1.0
    rho = 1.0
    if case.get("kind", DIFF) == MASS:
        rho = lognormal_kappa_q(nx, ny, nz, p, sigma2=0.1, seed=seed, device="cuda")
    return vc, kappa, rho


GAMMA_DT = (1.0 - 2.0 ** -0.5) * 1e-3  # the heat example's stage operator M + gamma dt K


def _coefs(kind):
    return (1.0, GAMMA_DT) if kind == MASS_DIFF else (1.0, 1.0)


def _box_operator(case, seed):
    vc, kappa, rho = _box_inputs(case, seed)
    kind = case.get("kind", DIFF)
    cm, ck = _coefs(kind)
    mesh = dict(nx=case["nx"], ny=case["ny"], nz=case["nz"], vcoord=vc)
    return femgpu.PAOperator(mesh, case["p"], kind, kappa=kappa, rho=rho, c_mass=cm, c_diff=ck)


def _box_plain(case, seed):
    vc, kappa, rho = _box_inputs(case, seed)
    kind = case.get("kind", DIFF)
    cm, ck = _coefs(kind)
    nx, ny, nz, p = case["nx"], case["ny"], case["nz"], case["p"]
    dofs, verts, ess = _box_maps(nx, ny, nz, p)
    if vc is None:
        vc = femgpu.unit_cube_vertices(nx, ny, nz)
    phi, grad, w, vg = _hex_element(p)
    E = dofs.shape[0]
    shape = lambda c: c if np.isscalar(c) else np.asarray(c).reshape(E, -1)  # noqa: E731
    return _Plain(dofs, len(ess), phi, grad, w, vg, vc[verts], kind, shape(kappa), shape(rho), cm, ck, ess)


def _vector(n, seed, dtype=torch.float64):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(n, generator=g, dtype=dtype, device="cuda")


def _native(x, NI, NJ, NK, NIp):
    out = torch.zeros((NK, NJ, NIp), dtype=x.dtype, device="cuda")
    out[:, :, :NI] = x.view(NK, NJ, NI)
    return out


def _stream():
    return torch.cuda.current_stream().cuda_stream


_CONN = [0, 1, 3, 2, 4, 5, 7, 6]  # (z, y, x) vertex order -> HexQ1 order


def _hex_inputs(case, seed):
    """The box's perturbed elements as a mesh generator hands them over: node coordinates, connectivity, DOF
    maps, coefficients."""
    dofs, verts, ess = _box_maps(case["nx"], case["ny"], case["nz"], case["p"])
    rng = np.random.default_rng(seed)
    vc = _vertices(case, rng)
    kind, q = case["kind"], (case["p"] + 1) ** 3
    E = dofs.shape[0]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    field = lambda s: torch.exp(s * torch.randn((E, q), generator=g, dtype=torch.float64, device="cuda")).cpu().numpy()  # noqa: E731
    kappa = field(0.5) if kind & DIFF else 1.0
    rho = field(0.2) if kind == MASS else 1.0
    return dofs, verts, ess, vc, kappa, rho


@functools.lru_cache(6)
def _tet_space(n, p):
    return tetmesh.unit_cube_space(n, p)


def _tet_inputs(case, seed):
    coords, dofs, nd, mask = _tet_space(case["n"], case["p"])
    rng = np.random.default_rng(seed)
    coords = coords.copy()
    inner = np.all((coords > 1e-12) & (coords < 1 - 1e-12), axis=1)
    coords[inner] += 0.2 / case["n"] * rng.uniform(-1, 1, size=(int(inner.sum()), 3))
    order, xi, phi, grad, w = _tet_element(case["p"], case["kind"])
    x0 = coords[dofs[:, 0]]
    pts = x0[:, None] + np.einsum("qd,edi->eqi", xi, coords[dofs[:, 1:4]] - x0[:, None])
    k = rng.normal(scale=4.0, size=(3, 3))
    ph = rng.uniform(0, 2 * np.pi, size=3)
    field = np.exp(np.sin(pts @ k.T + ph).sum(axis=-1) * 0.6)
    kappa = field if case["kind"] & DIFF else 1.0
    rho = 1.0 + 0.3 * np.cos(pts[..., 0] * 5.0) if case["kind"] & MASS else 1.0
    return coords, dofs, nd, mask, order, kappa, rho


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
_PRECOND = {"jacobi": femgpu.PC_JACOBI, "chebyshev": femgpu.PC_CHEBYSHEV, "none": femgpu.PC_NONE}


def _config(bits):
    return femgpu.SolverConfig(rtol=1e-11, max_iter=20000, precision=femgpu.FP32_IR if bits == 32 else femgpu.FP64)


def _load(n, ess, seed, dtype=torch.float64):
    """A random load or search direction: zero on the Dirichlet DOFs."""
    return _vector(n, seed, dtype).masked_fill(torch.as_tensor(ess, device="cuda"), 0.0)


def _batch_members(case):
    r = random.Random(case["sizes"])
    out = []
    for _ in range(case["count"]):
        n = [r.randint(case["lo"], case["hi"]) for _ in range(3)]
        out.append(dict(nx=n[0], ny=n[1], nz=n[2], p=r.choice([1, 2, 3]), geometry="uniform"))
    return out


def _network_inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    dims = (case["batch"], case["nz"], case["ny"], case["nx"])
    inp = torch.randn(dims + (2,), generator=g, device="cuda")
    target = torch.randn(dims, generator=g, device="cuda")
    parts = []
    for ci, co in _LAYERS:
        a = math.sqrt(6.0 / (27 * ci))
        parts += [a * (2 * torch.rand(co * 27 * ci, generator=g, device="cuda") - 1), 0.05 * torch.randn(co, generator=g, device="cuda")]
    return inp, target, torch.cat(parts)


def prepare(case, seed):
    family = case["family"]
    if family == "box":
        op = _box_operator(case, seed)
        if case["fmt"] == "affine":
            op.set_qdata_format(femgpu.QDATA_AFFINE)
        op.set_stream(_stream())
        dtype = torch.float64 if case["bits"] == 64 else torch.float32
        ess = _box_maps(case["nx"], case["ny"], case["nz"], case["p"])[2]
        x = _native(_load(op.n_dofs(), ess, seed + 1, dtype), op.NI, op.NJ, op.NK, op.NIp)
        return dict(op=op, x=x, y=torch.zeros_like(x), bits=case["bits"], family=family)
    if family == "hex":
        dofs, verts, ess, vc, kappa, rho = _hex_inputs(case, seed)
        cm, ck = _coefs(case["kind"])
        conn = verts[:, _CONN]
        maps = conn if case["p"] == 1 else dofs
        op = femgpu.HexMeshOperator(case["p"], vc, conn, maps, len(ess), case["kind"], kappa, rho, cm, ck,
                                    np.flatnonzero(ess))
        op.set_stream(_stream())
        dtype = torch.float64 if case["bits"] == 64 else torch.float32
        x = torch.zeros(op.native_len, dtype=dtype, device="cuda")
        x[:len(ess)] = _load(len(ess), ess, seed + 1, dtype)
        return dict(op=op, x=x, y=torch.zeros_like(x), bits=case["bits"], family=family)
    if family == "tet":
        coords, dofs, nd, mask, order, kappa, rho = _tet_inputs(case, seed)
        op = femgpu.TetOperator(case["p"], coords, dofs, nd, case["kind"], kappa, rho, *_coefs(case["kind"]),
                                quad_order=order, ess=mask)
        op.set_stream(_stream())
        x = _load(nd, mask.astype(bool), seed + 1)
        return dict(op=op, x=x, y=torch.zeros_like(x), bits=64, family=family)
    if family == "pcg":
        op = _box_operator(case, seed)
        op.set_stream(_stream())
        b = _load(op.n_dofs(), _box_maps(case["nx"], case["ny"], case["nz"], case["p"])[2], seed + 1)
        x = torch.zeros_like(b)
        if case["memory"] == "host":
            b, x = b.cpu().numpy(), x.cpu().numpy()
        return dict(op=op, b=b, x=x, cfg=_config(case["bits"]), precond=_PRECOND[case["precond"]], family=family)
    if family == "batch":
        ops, bs, xs = [], [], []
        for k, m in enumerate(_batch_members(case)):
            op = _box_operator(m, seed + 100 * k)
            op.set_qdata_format(femgpu.QDATA_AFFINE)
            op.set_stream(_stream())
            bs.append(_load(op.n_dofs(), _box_maps(m["nx"], m["ny"], m["nz"], m["p"])[2], seed + 100 * k + 1))
            xs.append(torch.zeros_like(bs[-1]))
            ops.append(op)
        return dict(ops=ops, bs=bs, xs=xs, cfg=_config(32), family=family)
    inp, target, params = _network_inputs(case, seed)
    net = femgpu.UNet()
    net.set_params(params.cpu().numpy())
    return dict(net=net, inp=inp, target=target, family=family)


def run(state):
    family = state["family"]
    if family in ("box", "hex", "tet"):
        x, y = state["x"], state["y"]
        apply = state["op"].apply_native if state["bits"] == 64 else state["op"].apply_native_f32
        apply(x.data_ptr(), y.data_ptr(), accumulate=False, constrained=True)
        return y
    if family == "pcg":
        x = state["x"]
        if isinstance(x, np.ndarray):
            x[:] = 0.0
        else:
            x.zero_()
        state["op"].pcg(state["b"], x, state["cfg"], state["precond"])
        return x
    if family == "batch":
        for x in state["xs"]:
            x.zero_()
        femgpu.batch_pcg(state["ops"], state["bs"], state["xs"], state["cfg"])
        return state["xs"]
    loss = state["net"].loss_grad(state["inp"], state["target"])
    return dict(loss=loss, grads=state["net"].get_grads())


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _hex_flops(p, kind):
    """Multiply-adds (x 2) of one sum-factorised element."""
    q = p + 1
    terms = (2 + 3 + 3 if kind & DIFF else 0) + (3 if kind == MASS else 1 if kind & MASS else 0)
    return 2 * (2 * q ** 4 * terms + q ** 3 * ((9 if kind & DIFF else 0) + (1 if kind & MASS else 0)))


def _box_work(c, bits, fmt, kind):
    E, n = c["nx"] * c["ny"] * c["nz"], math.prod(_grid(c["nx"], c["ny"], c["nz"], c["p"]))
    q = (c["p"] + 1) ** 3
    comps = {MASS: 1, DIFF: 6, MASS_DIFF: 7}[kind]
    words = q * comps
    if fmt == "affine":
        words = (6 if kind & DIFF else 0) + q * (2 if kind == MASS_DIFF else 1)
    return (E * words + 2 * n) * bits / 8, E * _hex_flops(c["p"], kind), n


def work(case):
    family = case["family"]
    if family == "box":
        b, f, _ = _box_work(case, case["bits"], case["fmt"], case["kind"])
        return dict(bytes=b, flops=f)
    if family == "hex":
        b, f, _ = _box_work(case, case["bits"], "full", case["kind"])
        E = case["nx"] * case["ny"] * case["nz"]
        return dict(bytes=b + 4 * E * (case["p"] + 1) ** 3, flops=f)
    if family == "tet":
        E, p, kind = 6 * case["n"] ** 3, case["p"], case["kind"]
        nl, n = {1: 4, 2: 10, 3: 20}[p], (case["n"] * p + 1) ** 3
        nq = len(_tet_element(p, kind)[4])
        words = (6 if kind & DIFF else 0)
        words += min(nq, {1: 0, 2: 10, 3: 35}[p]) if kind & DIFF else 0  # moments of the coefficient, or its points
        words += nq if kind & MASS else 0
        flops = 2 * nq * nl * ((6 if kind & DIFF else 0) + (2 if kind & MASS else 0))
        return dict(bytes=8 * (E * words + 2 * n) + 4 * E * nl, flops=E * flops)
    if family in ("pcg", "batch"):
        total = dict(bytes=0.0, flops=0.0)
        for m in ([case] if family == "pcg" else _batch_members(case)):
            cheb = family == "batch" or m["precond"] == "chebyshev"
            size = m["p"] * max(m["nx"], m["ny"], m["nz"])
            its, applies = (1.5 * size, 4) if cheb else (4.0 * size, 1)  # about what such problems take
            bits = 32 if family == "batch" else m["bits"]
            b, f, n = _box_work(m, bits, "affine" if family == "batch" else "full", DIFF)
            total["bytes"] += its * (applies * b + (8 if not cheb else 20) * n * bits / 8)
            total["flops"] += its * applies * f
        return total
    v = [case["batch"] * math.prod((case[k] - 1) // s + 1 for k in ("nz", "ny", "nx")) for s in (1, 2, 4)]
    level = [0, 0, 1, 1, 2, 2, 1, 0, 0]
    flops = sum(3 * 2 * 27 * ci * co * v[lv] for (ci, co), lv in zip(_LAYERS, level))
    return dict(bytes=2 * 3 * sum((ci + co) * v[lv] for (ci, co), lv in zip(_LAYERS, level)), flops=flops)


# ---------------------------------------------------------------------------
# the values in 64 bits
# ---------------------------------------------------------------------------
_LAYERS = [(2, 16), (16, 16), (16, 32), (32, 32), (32, 48), (48, 48), (80, 32), (48, 16), (16, 8)]


def _network_loss(inp, target, params):
    """Loss and gradients of the 3-level U-net in 64 bits."""
    F = torch.nn.functional
    params = params.double().requires_grad_(True)
    layers, o = [], 0
    for ci, co in _LAYERS:
        W = params[o:o + co * 27 * ci].view(co, 3, 3, 3, ci).permute(0, 4, 1, 2, 3)
        o += co * 27 * ci
        layers.append((W, params[o:o + co]))
        o += co
    k1 = torch.tensor([0.25, 0.5, 0.25], dtype=torch.float64, device="cuda")
    k3 = torch.einsum("z,y,x->zyx", k1, k1, k1)

    def conv(x, layer):
        return F.conv3d(x, layer[0], layer[1], padding=1)

    def down(x):
        return F.conv3d(x, k3.expand(x.shape[1], 1, 3, 3, 3), stride=2, padding=1, groups=x.shape[1])

    def up(x):
        return F.conv_transpose3d(x, 8 * k3.expand(x.shape[1], 1, 3, 3, 3), stride=2, padding=1, groups=x.shape[1])

    with torch.backends.cudnn.flags(enabled=False):
        x = inp.double().permute(0, 4, 1, 2, 3)
        h0 = conv(conv(x, layers[0]).relu(), layers[1]).relu()
        h1 = conv(conv(down(h0), layers[2]).relu(), layers[3]).relu()
        h2 = conv(conv(down(h1), layers[4]).relu(), layers[5]).relu()
        g1 = conv(torch.cat([up(h2), h1], dim=1), layers[6]).relu()
        g0 = conv(torch.cat([up(g1), h0], dim=1), layers[7]).relu()
        loss = (conv(g0, layers[8])[:, 0] - target.double()).square().mean()
        loss.backward()
    return dict(loss=float(loss), grads=params.grad)


def exact(case, seed):
    family = case["family"]
    if family == "box":
        NI, NJ, NK = _grid(case["nx"], case["ny"], case["nz"], case["p"])
        A = _box_plain(case, seed)
        x = _load(A.n, A.ess, seed + 1, torch.float64 if case["bits"] == 64 else torch.float32).double()
        return _native(A(x), NI, NJ, NK, -(-NI // 4) * 4)
    if family == "hex":
        dofs, verts, ess, vc, kappa, rho = _hex_inputs(case, seed)
        phi, grad, w, vg = _hex_element(case["p"])
        A = _Plain(dofs, len(ess), phi, grad, w, vg, vc[verts], case["kind"], kappa, rho, *_coefs(case["kind"]), ess)
        y = torch.zeros(-(-len(ess) // 4) * 4, dtype=torch.float64, device="cuda")
        y[:len(ess)] = A(_load(len(ess), ess, seed + 1, torch.float64 if case["bits"] == 64 else torch.float32).double())
        return y
    if family == "tet":
        coords, dofs, nd, mask, _, kappa, rho = _tet_inputs(case, seed)
        _, xi, phi, grad, w = _tet_element(case["p"], case["kind"])
        vg = np.broadcast_to(np.array([[-1, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]], dtype=float), (len(w), 4, 3))
        A = _Plain(dofs, nd, phi, grad, w, vg, coords[dofs[:, :4]], case["kind"], kappa, rho, *_coefs(case["kind"]),
                   mask.astype(bool))
        return A(_load(nd, mask.astype(bool), seed + 1))
    if family == "pcg":
        A = _box_plain(case, seed)
        x = A.solve(_load(A.n, A.ess, seed + 1))
        return x if case["memory"] == "device" else x.cpu().numpy()
    if family == "batch":
        out = []
        for k, m in enumerate(_batch_members(case)):
            if math.prod(_grid(m["nx"], m["ny"], m["nz"], m["p"])) > 300_000:
                out.append(None)  # a plain solve of this size takes too long
                continue
            A = _box_plain(m, seed + 100 * k)
            out.append(A.solve(_load(A.n, A.ess, seed + 100 * k + 1)))
        return out
    return _network_loss(*_network_inputs(case, seed))
