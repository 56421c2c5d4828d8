"""The work that users of this framework have it do, as measurable cases.

A case is one call (or the few calls) that a program's inner loop makes through the public
classes of `wavedg_b200`: Runge-Kutta steps of the wave system in FP64 and FP32, the operator
composition of the reference's examples, WaveHoltz periods alone and batched, the operators with
exact quadrature, the compressible Euler system, linear advection, and the training and prediction
step of the learned warm start.  `exact` restates each discretisation in plain FP64 torch: the mesh
and its connectivity, the bases and quadrature rules, the fluxes, the mass matrices and the
steppers are formed here and share nothing with the library.
"""
import math

import numpy as np
import torch

import wavedg_b200 as W
from wavedg_b200.dg import AdvectionSystem, EulerSystem, ExactDiscretisation, VariableAdvectionSystem, WaveHoltzBatch
from wavedg_b200.fno import FNO

DEV = "cuda"
F64 = torch.float64


# ------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the plain method as the 2D example runs it: a small uniform mesh, many short steps
        dict(name="rk4-32x32-p3", kind="rk4", nx=32, ny=32, n=4, mesh="uniform", bc="dirichlet", fp32=False, steps=10),
        # the drop-in composition of the examples (WaveEquation, WaveBC, MassMatrix::inv called one
        # by one) on an odd-sized mesh in file order (random numbering, every side pairing)
        dict(name="operators-61x47-p5", kind="operators", nx=61, ny=47, n=6, mesh="scrambled", bc="mixed"),
        # the headline throughput workload: 19.7 M DOF, bilinear elements, outflow, FP64 and FP32
        dict(name="rk4-512x512-p4", kind="rk4", nx=512, ny=512, n=5, mesh="perturbed", bc="outflow", fp32=False, steps=2),
        dict(name="rk4-512x512-p4-fp32", kind="rk4", nx=512, ny=512, n=5, mesh="perturbed", bc="outflow", fp32=True, steps=2),
        # one Helmholtz problem: the forced period that gives pi0, then one application of S
        dict(name="waveholtz-128x128-p4", kind="waveholtz", nx=128, ny=128, n=5, omega=20.0),
        # a batch of Helmholtz problems of uneven mesh, degree and frequency, one period each
        dict(name="batch-fp32-mixed", kind="batch", ne0=64, n0=4, om0=24.0, ne1=96, n1=5, om1=30.0, ne2=64, n2=7,
             om2=36.0, ne3=128, n3=4, om3=20.0),
        # approx_quad = false, the reference's default, stepped in time
        dict(name="exact-128x128-p4", kind="exactq", nx=128, ny=128, n=5, mesh="perturbed", bc="mixed", steps=2),
        # the Euler example with collocation and, as it ships, with exact quadrature
        dict(name="euler-256x256-p4", kind="euler", nx=256, ny=256, n=5, mesh="perturbed", approx=True, method="ssprk3", steps=1),
        dict(name="euler-exact-128x128-p4", kind="euler", nx=128, ny=128, n=5, mesh="perturbed", approx=False,
             method="ssprk3", steps=1),
        # the advection example: a rotating coefficient on a Gauss-Legendre basis, exact quadrature
        dict(name="advec2d-128x128-p4", kind="vadvect", nx=128, ny=128, n=5, mesh="perturbed", legendre=True, approx=False,
             method="ssprk3", steps=1),
        # a constant-coefficient hyperbolic system of two variables
        dict(name="advection-256x256-p4", kind="advect", nx=256, ny=256, n=5, nv=2, mesh="perturbed", steps=1),
        # one training step of the learned warm start's network at the shipped size
        dict(name="fno-train-512-b4", kind="fno", grid=512, width=32, modes=16, layers=4, hidden=64, batch=4, train=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh_size(rng, n, most):
    """An uneven nx x ny with at most `most` nodes."""
    cells = _log_int(rng, 64, max(65, most // (n * n)))
    nx = max(4, min(512, int(math.sqrt(cells) * rng.uniform(0.6, 1.5))))
    return nx, max(4, min(512, cells // nx))


def draw(rng):
    kind = rng.choice(["rk4", "rk4", "operators", "waveholtz", "batch", "exactq", "euler", "euler", "vadvect", "advect", "fno"])
    mesh = rng.choice(["uniform", "perturbed", "scrambled"])
    bc = rng.choice(["outflow", "dirichlet", "mixed"])
    if kind == "rk4":
        n = rng.choice([2, 3, 4, 5, 5, 6, 7, 8, 9])
        nx, ny = _mesh_size(rng, n, 6_000_000)
        return dict(kind=kind, nx=nx, ny=ny, n=n, mesh=mesh, bc=bc, fp32=rng.random() < 0.4, steps=rng.choice([1, 2, 5, 10]))
    if kind == "operators":
        n = rng.choice([2, 3, 4, 5, 6, 7, 8, 9])
        nx, ny = _mesh_size(rng, n, 2_000_000)
        return dict(kind=kind, nx=nx, ny=ny, n=n, mesh=mesh, bc=bc)
    if kind == "waveholtz":
        n = rng.choice([3, 4, 5, 7])
        ne = rng.choice([24, 33, 48, 64, 80]) if n < 7 else rng.choice([20, 32, 41])
        return dict(kind=kind, nx=ne, ny=ne, n=n, omega=round(rng.uniform(12.0, 40.0), 2))
    if kind == "batch":
        c = dict(kind=kind)
        for s in range(4):
            n = rng.choice([4, 5, 7])
            c.update({f"ne{s}": rng.choice([32, 48, 64, 80]) if n < 7 else rng.choice([24, 40, 48]), f"n{s}": n,
                      f"om{s}": round(rng.uniform(18.0, 40.0), 2)})
        return c
    if kind == "exactq":
        n = rng.choice([2, 3, 4, 5, 6, 7])
        nx, ny = _mesh_size(rng, n, 2_000_000 // n ** 2)
        return dict(kind=kind, nx=nx, ny=ny, n=n, mesh=mesh, bc=bc, steps=rng.choice([1, 2, 4]))
    if kind == "euler":
        approx = rng.random() < 0.5
        n = rng.choice([2, 3, 4, 5, 6, 7])
        nx, ny = _mesh_size(rng, n, 2_000_000 if approx else 2_000_000 // n ** 2)
        return dict(kind=kind, nx=nx, ny=ny, n=n, mesh=mesh, approx=approx, method=rng.choice(["ssprk3", "ssprk3", "rk4"]),
                    steps=rng.choice([1, 2]))
    if kind == "vadvect":
        n = rng.choice([2, 3, 4, 5, 6, 7])
        nx, ny = _mesh_size(rng, n, 1_000_000 // n ** 2)
        return dict(kind=kind, nx=nx, ny=ny, n=n, mesh=mesh, legendre=rng.random() < 0.6, approx=rng.random() < 0.35,
                    method=rng.choice(["ssprk3", "rk4"]), steps=rng.choice([1, 2]))
    if kind == "advect":
        n = rng.choice([2, 3, 4, 5, 6, 7, 8])
        nx, ny = _mesh_size(rng, n, 2_000_000)
        return dict(kind=kind, nx=nx, ny=ny, n=n, nv=rng.choice([1, 2, 3, 4]), mesh=mesh, steps=rng.choice([1, 2]))
    return dict(kind="fno", grid=rng.choice([128, 192, 256, 320, 384]), width=rng.choice([16, 32]), modes=rng.choice([8, 12, 16]),
                layers=rng.choice([2, 3, 4]), hidden=rng.choice([32, 64]), batch=rng.choice([1, 2, 3, 4]),
                train=rng.random() < 0.5)


# ------------------------------------------------------------------------------ meshes
def _mesh(kind, nx, ny, seed):
    """Vertices and quads of [-1, 1]^2: uniform; interior vertices moved by up to 0.2 h; the same in
    random element order with random corner rotations, as a mesh file would have it."""
    rng = np.random.default_rng([seed, nx, ny])
    x, y = np.meshgrid(-1 + 2 * np.arange(nx + 1) / nx, -1 + 2 * np.arange(ny + 1) / ny)
    v = np.stack([x, y], axis=-1)
    if kind != "uniform":
        d = rng.uniform(-0.2, 0.2, size=(ny - 1, nx - 1, 2))
        v[1:-1, 1:-1] += d * np.array([2 / nx, 2 / ny])
    v = v.reshape(-1, 2)
    i, j = np.meshgrid(np.arange(nx), np.arange(ny))
    a = (i + (nx + 1) * j).reshape(-1)
    q = np.stack([a, a + 1, a + nx + 2, a + nx + 1], axis=-1)
    if kind == "scrambled":
        q = q[rng.permutation(len(q))]
        q = np.take_along_axis(q, (np.arange(4)[None] + rng.integers(0, 4, size=(len(q), 1))) % 4, axis=1)
    return np.ascontiguousarray(v), np.ascontiguousarray(q.astype(np.int32))


def _codes(mid, bc):
    """Boundary codes (0 absorbing, 1 reflecting, 2 Dirichlet p = 0) of boundary edges by midpoint."""
    c = np.full(len(mid), {"outflow": 0, "dirichlet": 2, "mixed": 0}[bc], dtype=np.int32)
    if bc == "mixed":
        c[mid[:, 0] < -1 + 1e-9] = 1
        c[mid[:, 1] < -1 + 1e-9] = 2
    return c


# ------------------------------------------------------------------------------ 1D bases
def _legendre(n):
    return np.polynomial.legendre.leggauss(n)


def _lobatto(n):
    c = np.zeros(n)
    c[-1] = 1.0
    dc = np.polynomial.legendre.legder(c)
    x = np.concatenate([[-1.0], np.sort(np.polynomial.legendre.legroots(dc)) if n > 2 else [], [1.0]])
    ddc = np.polynomial.legendre.legder(dc)
    for _ in range(3 if n > 2 else 0):
        x[1:-1] -= np.polynomial.legendre.legval(x[1:-1], dc) / np.polynomial.legendre.legval(x[1:-1], ddc)
    x = 0.5 * (x - x[::-1])
    return x, 2.0 / (n * (n - 1) * np.polynomial.legendre.legval(x, c) ** 2)


def _interp(x, xq):
    """P[i, k] = phi_k(xq_i) of the Lagrange basis on x."""
    P = np.ones((len(xq), len(x)))
    for k in range(len(x)):
        for m in range(len(x)):
            if m != k:
                P[:, k] *= (xq - x[m]) / (x[k] - x[m])
    return P


def _deriv(x, xq):
    D = np.zeros((len(xq), len(x)))
    for k in range(len(x)):
        for a in range(len(x)):
            if a == k:
                continue
            p = np.full(len(xq), 1.0 / (x[k] - x[a]))
            for m in range(len(x)):
                if m not in (k, a):
                    p *= (xq - x[m]) / (x[k] - x[m])
            D[:, k] += p
    return D


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=DEV)


# ------------------------------------------------------------------------------ the discretisation in torch
SIDE_FROM, SIDE_TO = (0, 1, 3, 0), (1, 2, 2, 3)


class _Disc:
    """Nodal DG on the quads, states as (element, j, i, variable).  `rules`: None for collocation at
    the basis nodes, else the point counts of the volume, face and mass rules."""

    def __init__(self, verts, quads, n, legendre=False, rules=None):
        self.n, self.nel, self.exact = n, len(quads), rules is not None
        x, w = _legendre(n) if legendre else _lobatto(n)
        self.x = _t(x)
        corners = verts[quads]
        self.c = _t(corners)
        q, qf, qm = rules if rules else (n, n, n)
        xv, wv = _legendre(q) if rules else (x, w)
        xf, wf = _legendre(qf) if rules else (x, w)
        xm, wm = _legendre(qm) if rules else (x, w)
        eye = np.eye(n)
        self.P, self.D = _t(_interp(x, xv) if rules else eye), _t(_deriv(x, xv))
        self.Pf, self.wf = _t(_interp(x, xf) if rules else eye), _t(wf)
        self.e0, self.e1 = _t(_interp(x, np.array([-1.0]))[0]), _t(_interp(x, np.array([1.0]))[0])
        J = self._jac(_t(xv), _t(xv))
        Wq = _t(np.outer(wv, wv))[None]
        self.geo = [g * Wq for g in J]  # x_xi, y_xi, x_eta, y_eta times the weights at (eta, xi)
        Jm = self._jac(_t(xm), _t(xm))
        det = (Jm[0] * Jm[3] - Jm[1] * Jm[2]) * _t(np.outer(wm, wm))[None]
        if rules:
            B = _t(_interp(x, xm))
            BB = torch.einsum("qj,ri->qrji", B, B).reshape(qm * qm, n * n)
            M = torch.einsum("ep,pa,pb->eab", det.reshape(self.nel, -1), BB, BB)
            self.chol = torch.linalg.cholesky(M)
        else:
            self.minv = 1.0 / det[..., None]
        # sides: normals (outward for counter-clockwise corners), half lengths, midpoints, neighbours
        a, b = corners[:, SIDE_FROM, :], corners[:, SIDE_TO, :]
        d = b - a
        ln = np.hypot(d[..., 0], d[..., 1])
        sg = np.array([1.0, 1.0, -1.0, -1.0])
        self.nx, self.ny, self.meas = _t(sg * d[..., 1] / ln), _t(-sg * d[..., 0] / ln), _t(0.5 * ln)
        self.mid = 0.5 * (a + b)
        va, vb = quads[:, SIDE_FROM].astype(np.int64), quads[:, SIDE_TO].astype(np.int64)
        key = (np.minimum(va, vb) * (len(verts) + 1) + np.maximum(va, vb)).reshape(-1)
        order = np.argsort(key, kind="stable")
        pair = key[order][1:] == key[order][:-1]
        nb = np.full(key.size, -1, dtype=np.int64)
        nb[order[1:][pair]], nb[order[:-1][pair]] = order[:-1][pair], order[1:][pair]
        rev = (va.reshape(-1) != va.reshape(-1)[np.maximum(nb, 0)])
        k = np.arange(n)
        idx = np.maximum(nb, 0)[:, None] * n + np.where(rev[:, None], n - 1 - k[None], k[None])
        self.nb, self.nidx = _t((nb < 0).reshape(self.nel, 4)), _t(idx.reshape(-1))
        self.ends = [np.unique(ln).min()]

    def _jac(self, xi, eta):
        c = self.c[:, :, None, None, :]
        e, s = eta[:, None], xi[None, :]
        dxi = 0.25 * ((1 - e)[None, ..., None] * (c[:, 1] - c[:, 0]) + (1 + e)[None, ..., None] * (c[:, 2] - c[:, 3]))
        det = 0.25 * ((1 - s)[None, ..., None] * (c[:, 3] - c[:, 0]) + (1 + s)[None, ..., None] * (c[:, 2] - c[:, 1]))
        sh = (self.nel, len(eta), len(xi))
        return [g.expand(sh) for g in (dxi[..., 0], dxi[..., 1], det[..., 0], det[..., 1])]

    def nodes(self):
        e, s = self.x[:, None], self.x[None, :]
        c = self.c[:, :, None, None, :]
        sh = [0.25 * (1 - s) * (1 - e), 0.25 * (1 + s) * (1 - e), 0.25 * (1 + s) * (1 + e), 0.25 * (1 - s) * (1 + e)]
        return sum(f[None, ..., None] * c[:, k] for k, f in enumerate(sh))  # (element, j, i, 2)

    def at_points(self, u):
        return torch.einsum("qj,ri,ejid->eqrd", self.P, self.P, u) if self.exact else u

    def traces(self, u):
        return torch.stack([torch.einsum("j,ejid->eid", self.e0, u), torch.einsum("i,ejid->ejd", self.e1, u),
                            torch.einsum("j,ejid->eid", self.e1, u), torch.einsum("i,ejid->ejd", self.e0, u)], dim=1)

    def neighbours(self, T):
        return T.reshape(-1, T.shape[-1])[self.nidx].reshape(T.shape)

    def at_face_points(self, T):
        return torch.einsum("qk,eskd->esqd", self.Pf, T) if self.exact else T

    def volume(self, f, g):
        Xx, Yx, Xe, Ye = (v[..., None] for v in self.geo)
        F, G = Ye * f - Xe * g, -Yx * f + Xx * g
        if not self.exact:
            return torch.einsum("ri,ejrd->ejid", self.D, F) + torch.einsum("qj,eqid->ejid", self.D, G)
        return (torch.einsum("qj,ri,eqrd->ejid", self.P, self.D, F) + torch.einsum("qj,ri,eqrd->ejid", self.D, self.P, G))

    def lift(self, fh):
        """- sum over sides of the traces' transpose of the numerical flux at the face points."""
        h = fh * (self.wf[None, None, :, None] * self.meas[:, :, None, None])
        h = torch.einsum("qk,esqd->eskd", self.Pf, h) if self.exact else h
        return -(torch.einsum("j,eid->ejid", self.e0, h[:, 0]) + torch.einsum("i,ejd->ejid", self.e1, h[:, 1])
                 + torch.einsum("j,eid->ejid", self.e1, h[:, 2]) + torch.einsum("i,ejd->ejid", self.e0, h[:, 3]))

    def inv_mass(self, r):
        if not self.exact:
            return r * self.minv
        return torch.cholesky_solve(r.reshape(self.nel, self.n ** 2, -1), self.chol).reshape(r.shape)


def _wave_flux(q):
    z = torch.zeros_like(q[..., 0])
    return torch.stack([q[..., 1], q[..., 0], z], -1), torch.stack([q[..., 2], z, q[..., 0]], -1)


def _wave_rhs(d, codes, parts=("volume", "inner", "outer"), mass=True):
    """codes: (element, side) boundary codes; the right-hand side of the linear wave system."""
    nx, ny = d.nx[:, :, None], d.ny[:, :, None]
    code, bnd = codes[:, :, None, None], d.nb[:, :, None, None]

    def exterior(q):
        p, u, v = q[..., 0], q[..., 1], q[..., 2]
        out, tan = p + nx * u + ny * v, ny * u - nx * v
        ux, vx = ny * tan + 0.5 * nx * out, -nx * tan + 0.5 * ny * out
        absorb = torch.stack([nx * ux + ny * vx, ux, vx], -1)
        s, c = 2 * nx * ny, ny * ny - nx * nx
        reflect = torch.stack([p, c * u - s * v, -s * u - c * v], -1)
        return torch.where(code == 0, absorb, torch.where(code == 1, reflect, torch.stack([-p, u, v], -1)))

    def rhs(u):
        r = d.volume(*_wave_flux(d.at_points(u))) if "volume" in parts else 0.0
        T = d.traces(u)
        X = torch.where(bnd, exterior(T), d.neighbours(T))
        a, b = d.at_face_points(T), d.at_face_points(X)
        s, j = a + b, a - b
        nj = nx * j[..., 1] + ny * j[..., 2]
        fh = 0.5 * torch.stack([nx * s[..., 1] + ny * s[..., 2] + j[..., 0], nx * (s[..., 0] + nj), ny * (s[..., 0] + nj)], -1)
        r = r + d.lift(fh)
        return d.inv_mass(r) if mass else r

    return rhs


def _euler_rhs(d):
    def flux(q):
        rho, mx, my, E = q.unbind(-1)
        u, v = mx / rho, my / rho
        p = 0.4 * (E - 0.5 * rho * (u * u + v * v))
        return (torch.stack([mx, mx * u + p, mx * v, u * (E + p)], -1), torch.stack([my, mx * v, my * v + p, v * (E + p)], -1),
                torch.hypot(u, v) + torch.sqrt(1.4 * p / rho))

    nx, ny = d.nx[:, :, None, None], d.ny[:, :, None, None]

    def rhs(u):
        f, g, _ = flux(d.at_points(u))
        T = d.traces(u)
        X = torch.where(d.nb[:, :, None, None], T, d.neighbours(T))
        a, b = d.at_face_points(T), d.at_face_points(X)
        (fa, ga, sa), (fb, gb, sb) = flux(a), flux(b)
        fh = 0.5 * (nx * (fa + fb) + ny * (ga + gb) + torch.maximum(sa, sb)[..., None] * (a - b))
        return d.inv_mass(d.volume(f, g) + d.lift(fh))

    return rhs


def _advect_rhs(d, A):
    """Constant symmetric coefficients A = (A_0, A_1), upwind, zero outside."""
    nA = d.nx[:, :, None, None] * A[0] + d.ny[:, :, None, None] * A[1]
    ev, R = torch.linalg.eigh(nA.cpu())
    ab = (R * ev.abs()[..., None, :] @ R.transpose(-1, -2)).to(DEV)

    def rhs(u):
        T = d.traces(u)
        X = torch.where(d.nb[:, :, None, None], torch.zeros_like(T), d.neighbours(T))
        fh = 0.5 * (torch.einsum("esdc,eskc->eskd", nA, T + X) + torch.einsum("esdc,eskc->eskd", ab, T - X))
        return d.inv_mass(d.volume(u @ A[0].T, u @ A[1].T) + d.lift(fh))

    return rhs


def _vadvect_rhs(d, a):
    """One variable with the nodal coefficient a (element, j, i, 2), upwind, zero outside."""
    ap = d.at_points(a)
    Ta = d.traces(a)
    nrm = torch.stack([d.nx, d.ny], -1)[:, :, None, :]
    own = (d.at_face_points(Ta) * nrm).sum(-1, keepdim=True)
    nbr = (d.at_face_points(d.neighbours(Ta)) * nrm).sum(-1, keepdim=True)
    inner = (~d.nb)[:, :, None, None]

    def rhs(u):
        U, T = d.at_points(u), d.traces(u)
        a0, b0 = d.at_face_points(T), d.at_face_points(d.neighbours(T))
        fh = 0.5 * (own + own.abs()) * a0 + inner * 0.5 * (nbr - nbr.abs()) * b0
        return d.inv_mass(d.volume(U * ap[..., :1], U * ap[..., 1:]) + d.lift(fh))

    return rhs


RK_A = (0.0, -567301805773.0 / 1357537059087.0, -2404267990393.0 / 2016746695238.0, -3550918686646.0 / 2091501179385.0,
        -1275806237668.0 / 842570457699.0)
RK_B = (1432997174477.0 / 9575080441755.0, 5161836677717.0 / 13612068292357.0, 1720146321549.0 / 2090206949498.0,
        3134564353537.0 / 4481467310338.0, 2277821191437.0 / 14882151754819.0)
RK_C = (0.0, 1432997174477.0 / 9575080441755.0, 2526269341429.0 / 6820363962896.0, 2006345519317.0 / 3224310063776.0,
        2802321613138.0 / 2924317926251.0)


def _advance(rhs, u, dt, steps, method="rk4", t=0.0, force=None):
    for _ in range(steps):
        if method == "ssprk3":
            y = u + dt * rhs(u)
            y = 0.25 * (3 * u + y + dt * rhs(y))
            u = (u + 2 * y + 2 * dt * rhs(y)) / 3
        else:
            k = torch.zeros_like(u)
            for a, b, c in zip(RK_A, RK_B, RK_C):
                r = rhs(u)
                if force is not None:
                    r = r + force(t + c * dt)
                k = a * k + dt * r
                u = u + b * k
        t += dt
    return u


# ------------------------------------------------------------------------------ inputs
def _gauss(xy, seed, count, lo=0.03, hi=0.1):
    """A sum of seeded Gaussian pulses at points (..., 2)."""
    r = np.random.default_rng([seed, count, 7])
    out = torch.zeros(xy.shape[:-1], dtype=F64, device=DEV)
    for cx, cy, s, a in zip(r.uniform(-0.8, 0.8, count), r.uniform(-0.8, 0.8, count), r.uniform(lo, hi, count),
                            r.standard_normal(count)):
        out += a * torch.exp(-((xy[..., 0] - cx) ** 2 + (xy[..., 1] - cy) ** 2) / (2 * s * s))
    return out


def _state(case, d, seed):
    """Initial states: pressure and velocity pulses; for Euler, smooth subsonic variations of a gas."""
    xy = d.nodes()
    if case["kind"] == "euler":
        b = [torch.tanh(_gauss(xy, seed + k, 6, 0.1, 0.3)) for k in range(4)]
        rho, u, v, p = 1 + 0.1 * b[0], 0.1 * b[1], 0.1 * b[2], 1 + 0.1 * b[3]
        return torch.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)], -1)
    nv = {"vadvect": 1, "advect": case.get("nv", 1)}.get(case["kind"], 3)
    return torch.stack([_gauss(xy, seed + 100 * k, 8) for k in range(nv)], -1)


def _dt(case):
    """The examples' time step 0.1 h / (P + 1)^2."""
    return 0.1 * min(2.0 / case["nx"], 2.0 / case["ny"]) / case["n"] ** 2


def _rules(case):
    n, k = case["n"], case["kind"]
    if k == "exactq":  # degrees 2 n - 2 in the volume, 2 n on faces and in the mass matrix
        return 1 + (2 * n - 2) // 2, 1 + 2 * n // 2, 1 + 2 * n // 2
    if k == "euler" and not case["approx"]:
        return 2 * n, 2 * n, n + 1
    if k == "vadvect" and not case["approx"]:
        return 1 + (3 * n - 3) // 2, 1 + (3 * n - 1) // 2, n + 1
    return None


def _disc(case, seed):
    v, q = _mesh(case.get("mesh", "uniform"), case["nx"], case["ny"], seed)
    return v, q, _Disc(v, q, case["n"], bool(case.get("legendre")), _rules(case))


def _matrices(nv, seed):
    """Two seeded symmetric coefficient matrices of order one."""
    r = np.random.default_rng([seed, nv, 11]).standard_normal((2, nv, nv)) / math.sqrt(nv)
    return 0.5 * (r + r.transpose(0, 2, 1)) + np.array([1.0, 0.5])[:, None, None] * np.eye(nv)


def _forcing(case, seed):
    """omega^2 exp(-|x - x0|^2 / (2 0.05^2)) against the basis with n Gauss points, pressure only."""
    v, q = _mesh("uniform", case["nx"], case["ny"], seed)
    d = _Disc(v, q, case["n"])
    g, w = _legendre(case["n"])
    x0 = np.random.default_rng([seed, 3]).uniform(-0.5, 0.5, 2)
    B = _t(_interp(_lobatto(case["n"])[0], g))
    e, s = _t(g)[:, None], _t(g)[None, :]
    c = d.c[:, :, None, None, :]
    sh = [0.25 * (1 - s) * (1 - e), 0.25 * (1 + s) * (1 - e), 0.25 * (1 + s) * (1 + e), 0.25 * (1 - s) * (1 + e)]
    xy = sum(f[None, ..., None] * c[:, k] for k, f in enumerate(sh))
    J = d._jac(_t(g), _t(g))
    f = torch.exp(-((xy[..., 0] - x0[0]) ** 2 + (xy[..., 1] - x0[1]) ** 2) / (2 * 0.05 ** 2)) * case["omega"] ** 2
    p = torch.einsum("qj,ri,eqr->eji", B, B, f * (J[0] * J[3] - J[1] * J[2]) * _t(np.outer(w, w)))
    z = torch.zeros_like(p)
    return d, torch.stack([p, z, z], -1)


def _solves(case):
    return [dict(nx=case[f"ne{s}"], ny=case[f"ne{s}"], n=case[f"n{s}"], omega=case[f"om{s}"]) for s in range(4)]


def _fno_data(case, seed):
    """Seeded parameters with the spread that training starts from, inputs (forcing, omega, x, y) and targets."""
    r = np.random.default_rng([seed, 5])
    C, H, M, G = case["width"], case["hidden"], 2 * case["modes"] ** 2, case["grid"]

    def U(shape, s):
        return (r.random(shape, dtype=np.float32) * 2 - 1) * np.float32(s)

    p = {"P_w": U((C, 4), 0.5), "P_b": U((C,), 0.5), "Q1_w": U((H, C), C ** -0.5), "Q1_b": U((H,), C ** -0.5),
         "Q2_w": U((3, H), H ** -0.5), "Q2_b": U((3,), H ** -0.5)}
    for k in range(case["layers"]):
        p[f"R{k}"], p[f"W{k}"], p[f"b{k}"] = U((C, C, M, 2), 1.0 / C ** 1.5), U((C, C), C ** -0.5), U((C,), C ** -0.5)
    x = (torch.arange(G, device=DEV, dtype=F64) + 0.5) * 2 / G - 1
    xx, yy = x[None, :].expand(G, G), x[:, None].expand(G, G)
    inp, tgt = [], []
    for b in range(case["batch"]):
        cx, cy = r.uniform(-0.5, 0.5, 2)
        r2 = (xx - cx) ** 2 + (yy - cy) ** 2
        inp.append(torch.stack([torch.exp(-r2 / 0.005), torch.ones_like(xx), xx, yy]))
        s = torch.sqrt(r2 + 0.01)
        tgt.append(torch.stack([torch.cos(20 * s), torch.sin(20 * s) * (xx - cx) / s, torch.sin(20 * s) * (yy - cy) / s]))
    return p, torch.stack(inp).float().contiguous(), torch.stack(tgt).float().contiguous()


class _Resident:
    """The handle's resident single-precision state as an array on the device."""

    def __init__(self, system):
        self.system = system
        self.__cuda_array_interface__ = dict(shape=(system.ndof,), typestr="<f4", data=(system.state_ptr(), False), version=3)


# ------------------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    kind = case["kind"]
    if kind == "fno":
        p, inp, tgt = _fno_data(case, seed)
        net = FNO(grid=case["grid"], width=case["width"], modes=case["modes"], layers=case["layers"], hidden=case["hidden"])
        net.load_state_dict(p)
        return dict(case=case, net=net, inp=inp, tgt=tgt)
    if kind == "waveholtz":
        v, q = _mesh("uniform", case["nx"], case["ny"], seed)
        mesh = W.Mesh2D.from_vertices(v, q)
        wh = W.WaveHoltz(case["omega"], mesh, case["n"], np.zeros(mesh.n_edges(1), dtype=np.int32), approx_quad=True)
        F = _forcing(case, seed)[1].reshape(-1).contiguous()
        return dict(case=case, wh=wh, F=F, w=torch.zeros_like(F))
    if kind == "batch":
        systems, F = [], []
        for k, c in enumerate(_solves(case)):
            v, q = _mesh("uniform", c["nx"], c["ny"], seed)
            mesh = W.Mesh2D.from_vertices(v, q)
            systems.append(W.WaveSystem(mesh, c["n"], np.zeros(mesh.n_edges(1), dtype=np.int32), precision="fp32"))
            F.append(_forcing(c, seed + k)[1].reshape(-1).contiguous())
        b = WaveHoltzBatch(systems, [c["omega"] for c in _solves(case)])
        return dict(case=case, batch=b, F=F, W=[torch.zeros_like(f) for f in F])
    v, q = _mesh(case["mesh"], case["nx"], case["ny"], seed)
    d = _Disc(v, q, case["n"], bool(case.get("legendre")))
    u = _state(case, d, seed).reshape(-1).contiguous()
    mesh = W.Mesh2D.from_vertices(v, q)
    s = dict(case=case, u=u, dt=_dt(case))
    if kind in ("rk4", "operators", "exactq"):
        codes = _codes(mesh.boundary_midpoints(), case["bc"])
    if kind == "rk4":
        s["sys"] = W.WaveSystem(mesh, case["n"], codes, precision="fp32" if case["fp32"] else "fp64")
        if case["fp32"]:
            s["sys"].upload(u)
            s["out"] = torch.as_tensor(_Resident(s["sys"]), device=DEV)
    elif kind == "operators":
        basis = W.QuadratureRule.quadrature_rule(case["n"], W.QuadratureRule.GaussLobatto)
        s.update(eq=W.WaveEquation(mesh, basis, True), bc=W.WaveBC(mesh, codes, basis, True), mass=W.MassMatrix(mesh, basis),
                 du=torch.zeros_like(u))
    elif kind == "exactq":
        s["sys"] = ExactDiscretisation(mesh, case["n"], codes)
    elif kind == "euler":
        s["sys"] = EulerSystem(mesh, case["n"], approx_quad=case["approx"])
    elif kind == "advect":
        a = _matrices(case["nv"], seed)
        s["sys"] = AdvectionSystem(case["nv"], mesh, case["n"], a.transpose(0, 2, 1).reshape(-1))
    elif kind == "vadvect":
        basis = W.QuadratureRule.quadrature_rule(case["n"], W.QuadratureRule.GaussLegendre if case["legendre"]
                                                 else W.QuadratureRule.GaussLobatto)
        s["sys"] = VariableAdvectionSystem(1, mesh, basis, _rotation(d).cpu().numpy(), case["approx"])
    return s


def _rotation(d):
    xy = d.nodes()
    return torch.stack([-xy[..., 1], xy[..., 0]], -1).contiguous()


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "rk4":
        if case["fp32"]:
            s["sys"].step_state(s["dt"], 0.0, case["steps"])
            return s["out"]
        s["sys"].rk4_steps(s["u"], s["dt"], 0.0, case["steps"])
        return s["u"]
    if kind == "operators":
        s["du"].zero_()
        s["eq"].action(s["u"], s["du"])
        s["bc"].action(s["u"], s["du"])
        s["mass"].inv(3, s["du"])
        return s["du"]
    if kind == "waveholtz":
        s["wh"].pi0(s["w"], s["F"])
        pi0 = s["w"].clone()
        s["wh"].S(s["w"])
        return [pi0, s["w"]]
    if kind == "batch":
        return s["batch"].solve(s["F"], tol=1e-6, maxit=1, W=s["W"])[0]
    if kind in ("exactq", "advect"):
        s["sys"].rk4_steps(s["u"], s["dt"], 0.0, case["steps"])
        return s["u"]
    if kind in ("euler", "vadvect"):
        s["sys"].steps(s["u"], s["dt"], 0.0, case["steps"], case["method"])
        return s["u"]
    net = s["net"]
    if not case["train"]:
        return net.forward(s["inp"])
    y = net.forward(s["inp"], keep=True)
    loss, dy = net.mse(y, s["tgt"])
    net.backward(dy)
    return dict(y=y, loss=loss, **net.grads)


# ------------------------------------------------------------------------------ work
def _dg_flops(n, nv, q, qf, point, face):
    """Per element and right-hand side: interpolation to q x q points and back (none when q is n),
    the two derivative contractions, `point` flops a volume point, `face` a face point."""
    up = 2 * nv * (q * n * n + q * q * n) if q != n else 0
    back = 4 * nv * (q * q * n + q * n * n) if q != n else 4 * nv * n ** 3
    faces = 4 * (qf * face + (6 * nv * qf * n if qf != n else 0))
    return up + back + q * q * point + faces + n * n * (4 * nv + 10)


def work(case):
    kind = case["kind"]
    if kind == "fno":
        # the grid's activations once in and once out of each pointwise layer in 16 bits, the spectral
        # weights in 32; forward, and twice that for the backward pass
        P, C, B = case["grid"] ** 2, case["width"], case["batch"]
        act = B * P * (4 * 4 + 3 * 4 + 2 * C * 2 * (case["layers"] + 1))
        spec = case["layers"] * C * C * 2 * case["modes"] ** 2 * 8
        fl = B * P * 2 * (4 * C + case["layers"] * (C * C + 4 * C * case["modes"] * 2) + C * case["hidden"] + 3 * case["hidden"])
        k = 3 if case["train"] else 1
        return dict(bytes=k * (act + spec), flops=k * fl)
    if kind == "batch":
        w = [work(dict(c, kind="waveholtz")) for c in _solves(case)]
        return dict(bytes=sum(x["bytes"] for x in w) / 4, flops=sum(x["flops"] for x in w) / 2)
    nel, n = case["nx"] * case["ny"], case["n"]
    nv = {"euler": 4, "vadvect": 1, "advect": case.get("nv", 1)}.get(kind, 3)
    val = 4 if case.get("fp32") else 8
    state, geo = nel * nv * n * n * val, 64 * nel
    q, qf, _ = _rules(case) or (n, n, n)
    point, face = {"euler": (50, 110), "advect": (8 * nv * nv, 8 * nv * nv), "vadvect": (8, 10)}.get(kind, (20, 25))
    fl = nel * _dg_flops(n, nv, q, qf, point, face)
    if kind == "operators":
        return dict(bytes=2 * state + geo, flops=fl)
    if kind == "waveholtz":
        periods, nt = 2, math.ceil(2 * math.pi / case["omega"] / (0.5 * 2.0 / case["nx"] / n ** 2))
        return dict(bytes=4 * state + geo, flops=periods * 5 * nt * fl)
    stages = case["steps"] * (3 if case.get("method") == "ssprk3" else 5)
    # a state that the chip can hold is read and written once; a larger one streams through every
    # stage with its register (or, for SSPRK3, with the step's first state)
    once = 3 * state < 120e6
    extra = 2 * q * q * 8 * nel + 8 * qf * 8 * nel if kind == "vadvect" else 0
    moved = 2 * state + geo + extra if once else stages * ((4 if stages % 5 == 0 else 3) * state + geo + extra) - state
    return dict(bytes=moved, flops=stages * fl)


# ------------------------------------------------------------------------------ exact
def _side_codes(d, bc):
    c = _codes(d.mid.reshape(-1, 2), bc).reshape(d.nel, 4)
    return _t(c)


def _wh_exact(case, seed, unforced):
    """pi0 of the forcing (and S pi0): nt steps a period, the filter dt K(t) at the step times."""
    d, F = _forcing(case, seed)
    om, n = case["omega"], case["n"]
    rhs = _wave_rhs(d, _side_codes(d, "outflow"))
    T = 2 * math.pi / om
    nt = math.ceil(T / (0.5 * (2.0 / case["nx"]) / n ** 2))
    dt = T / nt
    K = lambda t: om / math.pi * (math.cos(om * t) - 0.25)  # noqa: E731
    MF = d.inv_mass(F)

    def period(u, acc, force):
        t = 0.0
        for it in range(1, nt + 1):
            u = _advance(rhs, u, dt, 1, "rk4", t, force)
            t += dt
            acc = acc + (0.5 if it == nt else 1.0) * dt * K(t) * u
        return acc

    z = torch.zeros_like(F)
    pi0 = period(z, z, lambda t: (-math.sin(om * t) / om) * MF)
    if not unforced:
        return pi0.reshape(-1)
    return [pi0.reshape(-1), period(pi0, 0.5 * dt * K(0.0) * pi0, None).reshape(-1)]


def _fno_exact(case, seed):
    p, inp, tgt = _fno_data(case, seed)
    P = {k: torch.as_tensor(v, device=DEV).double().requires_grad_(case["train"]) for k, v in p.items()}
    G, m, C = case["grid"], case["modes"], case["width"]
    x = inp.double()
    B = len(x)

    def mix(w, b, v):
        return torch.einsum("oc,bcxy->boxy", w, v) + b[None, :, None, None]

    def gelu(z):
        return 0.5 * z * (1 + torch.erf(z * math.sqrt(0.5)))

    v = mix(P["P_w"], P["P_b"], x)
    for k in range(case["layers"]):
        h = torch.fft.rfft2(v)
        R = torch.view_as_complex(P[f"R{k}"]).reshape(C, C, 2 * m, m)
        lo = torch.einsum("bcyx,coyx->boyx", h[:, :, :m, :m], R[:, :, :m])
        hi = torch.einsum("bcyx,coyx->boyx", h[:, :, -m:, :m], R[:, :, m:])
        mid = torch.zeros(B, C, G - 2 * m, m, dtype=lo.dtype, device=DEV)
        full = torch.cat([torch.cat([lo, mid, hi], 2), torch.zeros(B, C, G, G // 2 + 1 - m, dtype=lo.dtype, device=DEV)], 3)
        z = torch.fft.irfft2(full, s=(G, G)) + mix(P[f"W{k}"], P[f"b{k}"], v)
        v = gelu(z) if k < case["layers"] - 1 else z
    y = mix(P["Q2_w"], P["Q2_b"], gelu(mix(P["Q1_w"], P["Q1_b"], v)))
    if not case["train"]:
        return y
    e = y - tgt.double()
    (e * e).mean().backward()
    return dict(y=y.detach(), loss=None, **{k: t.grad for k, t in P.items()})


def exact(case, seed):
    kind = case["kind"]
    if kind == "fno":
        return _fno_exact(case, seed)
    with torch.no_grad():
        if kind == "waveholtz":
            return _wh_exact(case, seed, True)
        if kind == "batch":
            return [_wh_exact(c, seed + k, False) for k, c in enumerate(_solves(case))]
        _, _, d = _disc(case, seed)
        u = _state(case, d, seed)
        if kind == "operators":
            return _wave_rhs(d, _side_codes(d, case["bc"]))(u).reshape(-1)
        if kind in ("rk4", "exactq"):
            rhs = _wave_rhs(d, _side_codes(d, case["bc"]))
            u = u.float().double() if case.get("fp32") else u
        elif kind == "euler":
            rhs = _euler_rhs(d)
        elif kind == "advect":
            rhs = _advect_rhs(d, _t(_matrices(case["nv"], seed)))
        else:
            rhs = _vadvect_rhs(d, _rotation(d))
        return _advance(rhs, u, _dt(case), case["steps"], case.get("method", "rk4")).reshape(-1)
