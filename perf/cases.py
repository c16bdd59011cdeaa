"""The work that users of the framework have it do, as measurable cases.

A case is a dict of plain values; ``kind`` names the entry point it goes through:

  run       Quadesth.run: assembly, solve, reorganisation, boundary stresses and internal
            points of one boundary-value problem (main.f90:38-68), results on the host
  system    the phase calls of the same sequence without post-processing (geometry,
            ghmat8, solve, reorganize): the loop of a parameter study
  assembly  geometry and ghmat8 alone, A and FI left on the device
  points    Somigliana displacements and stresses of a solved problem at many points, on
            device-resident arrays or on host arrays
  batch     many small boxes with eight load cases each, assembled and solved together
  adjoint   objective and its gradient in shape and material (forward and backward)
  dense     a caller's own dense system on host buffers, by dgesv or solve_system

Boxes are kx x ky x kz quad9 elements along the edges with nearly square elements, either
on rollers with three pins and a uniform top traction in a random direction or clamped at
x = 0; sides, material and loads come from the seed.  ``exact`` restates the discrete
problem in plain torch FP64.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from bem3d_elastostatic_b200 import _lib, adjoint
from bem3d_elastostatic_b200.api import Batch, Quadesth, dgesv, solve_system
from bem3d_elastostatic_b200.mesh import Mesh, box_mesh, hollow_sphere, loaded_box


def listed():
    return [
        # the smallest benchmark problem (cube with 2 x 2 elements a face): all latency
        dict(name="run_294dof", kind="run", kx=2, ky=2, kz=2, clamped=False, precision="fp64", points=27),
        # the size of the reference's shipped input: 2,598 DOF and 1,965 internal points
        dict(name="run_2598dof", kind="run", kx=6, ky=6, kz=6, clamped=False, precision="fp64", points=1965),
        # a clamped plate in plain FP64, the default precision: the DGESV replacement
        dict(name="plate_fp64", kind="system", kx=20, ky=20, kz=2, clamped=True, precision="fp64"),
        # an ordinary ragged box in the first mixed mode
        dict(name="box_fp32ir", kind="system", kx=11, ky=8, kz=13, clamped=False, precision="fp32-ir"),
        # the 16 x 16 cube (18,438 DOF) in the fast mixed mode
        dict(name="cube16_bf16ir", kind="system", kx=16, ky=16, kz=16, clamped=False, precision="bf16-ir"),
        # the largest: 56,454 DOF in the fast mixed mode
        dict(name="cube28_bf16ir", kind="system", kx=28, ky=28, kz=28, clamped=False, precision="bf16-ir"),
        # assembly by itself with the FP32 far-field option, kept on the device
        dict(name="assembly_fp32far", kind="assembly", kx=14, ky=17, kz=12, clamped=False, precision="fp32-far"),
        # a plate's stress field at many points, device-resident
        dict(name="points_100k", kind="points", kx=20, ky=20, kz=2, clamped=True, points=100_003, host=False),
        # a few thousand probe points through the host interface
        dict(name="points_3k_host", kind="points", kx=9, ky=8, kz=10, clamped=False, points=3001, host=True),
        # many small systems with eight load cases each
        dict(name="batch_96", kind="batch", count=96, precision="fp32-ir"),
        # shape and material gradient on a hollow sphere: forward, transposed solve, backward
        dict(name="adjoint_sphere8", kind="adjoint", m=8),
        # the DGESV drop-in on host buffers, general dense matrix, four right-hand sides
        dict(name="dgesv_1500", kind="dense", n=1500, nrhs=4, how="dgesv"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _edges(rng, lo, hi):
    """kx, ky, kz of a box with about E surface elements, E log-uniform in [lo, hi]."""
    k = math.sqrt(_log_int(rng, lo, hi) / 6.0)
    r = [rng.uniform(0.7, 1.4) for _ in range(3)]
    s = math.sqrt(3.0 / (r[0] * r[1] + r[1] * r[2] + r[2] * r[0]))
    return dict(zip(("kx", "ky", "kz"), (max(1, math.floor(k * s * f + 0.5)) for f in r)))


def draw(rng):
    kind = rng.choice(["run", "system", "system", "assembly", "points", "batch", "adjoint", "dense"])
    clamped = rng.random() < 0.5
    if kind == "run":
        return dict(kind=kind, **_edges(rng, 12, 500), clamped=clamped, precision="fp64", points=_log_int(rng, 20, 4000))
    if kind == "system":
        prec, top = rng.choice([("fp64", 900), ("fp32-ir", 2400), ("bf16-ir", 4000)])
        return dict(kind=kind, **_edges(rng, 24, top), clamped=clamped, precision=prec)
    if kind == "assembly":
        return dict(kind=kind, **_edges(rng, 24, 2000), clamped=clamped, precision=rng.choice(["fp64", "fp32-far"]))
    if kind == "points":
        return dict(kind=kind, **_edges(rng, 54, 900), clamped=clamped, points=_log_int(rng, 100, 100_000),
                    host=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, count=_log_int(rng, 8, 96), precision=rng.choice(["fp32-ir", "fp64"]))
    if kind == "adjoint":
        return dict(kind=kind, m=rng.randint(2, 8))
    how = rng.choice(["dgesv", "fp64", "fp32-ir"])
    return dict(kind=kind, n=_log_int(rng, 150, 3000), nrhs=rng.randint(1, 6) if how == "dgesv" else 1, how=how)


# ----------------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------------

def _box(case, seed) -> Mesh:
    rng = np.random.default_rng(seed)
    k = np.array([case["kx"], case["ky"], case["kz"]])
    side = k / k.max() * rng.uniform(0.85, 1.2, 3)
    coords, kconec, faces = box_mesh(*side, *(int(v) for v in k))
    ne = kconec.shape[1]
    nu, young = rng.uniform(0.1, 0.42), 1.0
    kode = np.ones((ne, 3), dtype=np.int32)
    bc = np.zeros((ne, 9, 3))
    load = rng.standard_normal(3)
    if case["clamped"]:
        kode[faces == "x0"] = 0
        pins = []
    else:
        kode[faces == "z0", 2] = 0
        at = lambda p: int(np.argmin(np.abs(coords - p).max(1)))  # noqa: E731
        i0, i1 = at((0.0, 0.0, 0.0)), at((side[0], 0.0, 0.0))
        pins = [3 * i0, 3 * i0 + 1, 3 * i1 + 1]
    bc[faces == "z1"] = load
    pts = np.zeros((0, 3))
    if case.get("points"):
        pts = side * rng.uniform(0.05, 0.95, (case["points"], 3))
    return Mesh(coords[:, 0], coords[:, 1], coords[:, 2], np.full(ne, 9), kconec, kode.reshape(-1),
                bc.reshape(ne, 27).T, young / (2.0 * (1.0 + nu)), nu, pts[:, 0], pts[:, 1], pts[:, 2], pins=pins)


def _sphere(case, seed) -> Mesh:
    rng = np.random.default_rng(seed)
    return hollow_sphere(case["m"], a=1.0, b=rng.uniform(1.6, 2.4), nu=rng.uniform(0.1, 0.42),
                         pressure=rng.uniform(0.5, 2.0))


def _boxes(case, seed):
    """Boxes of every size from 1 to 6 elements an edge in turn, with eight top tractions each."""
    rng = np.random.default_rng(seed)
    return [loaded_box(*rng.uniform(0.5, 2.0, 3), i % 6 + 1, rng.uniform(0.05, 0.45), 1.0, rng.standard_normal((8, 3)))
            for i in range(case["count"])]


def _dense(case, seed):
    rng = np.random.default_rng(seed)
    n = case["n"]
    A = rng.standard_normal((n, n))
    if case["how"] != "dgesv":  # solve_system's systems are diagonally weighted, as collocation systems are
        A = A / math.sqrt(n) + 3.0 * np.eye(n)
    return np.asfortranarray(A), np.asfortranarray(rng.standard_normal((n, case["nrhs"])))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "dense":
        A, B = _dense(case, seed)
        return dict(case=case, A=A, B=B, ctx=_lib.Context(0))
    if kind == "batch":
        b = Batch(0)
        for mesh, bcs in _boxes(case, seed):
            b.add(mesh, bcs)
        return dict(case=case, batch=_Owned(b))
    mesh = _sphere(case, seed) if kind == "adjoint" else _box(case, seed)
    st = dict(case=case, mesh=mesh, q=Quadesth(mesh))
    if kind == "points":
        q = st["q"]
        q.precompute_element_geometry()
        q.ghmat8()
        q.solve_linear_system("fp64")
        q.reorganize_solution()
        if not case["host"]:
            l = mesh.l  # noqa: E741 - reference name
            st["in"] = [torch.tensor(v, device="cuda") for v in (mesh.cx, mesh.cy, mesh.cz)]
            st["out"] = [torch.empty(l, c, dtype=torch.float64, device="cuda") for c in (3, 6, 3, 1)]
            torch.cuda.synchronize()
    return st


class _Owned:
    """A batch that is closed with its last reference, as a program's own object would be."""

    def __init__(self, batch):
        self.b = batch

    def __del__(self):
        self.b.close()


class _DeviceArray:
    """A device address as an array for torch; `owner` keeps the memory alive."""

    def __init__(self, ptr, shape, strides, owner):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, strides=strides, typestr="<f8", data=(ptr, False), version=3)


# ----------------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------------

def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "run":
        res = st["q"].run(case["precision"])
        return {k: v for k, v in res.items() if k != "solve_info"}
    if kind == "system":
        q = st["q"]
        q.precompute_element_geometry()
        q.ghmat8()
        x = q.solve_linear_system(case["precision"])
        u, t = q.reorganize_solution()
        return {"x": x, "u": u, "t": t}
    if kind == "assembly":
        q = st["q"]
        q.precompute_element_geometry()
        q.ghmat8(case["precision"])
        A, lda, FI = _lib.C.c_void_p(), _lib.C.c_int64(), _lib.C.c_void_p()
        q.ctx.check(q.ctx.L.bem_device_state(q.ctx.h, _lib.C.byref(A), _lib.C.byref(lda), _lib.C.byref(FI), None),
                    "device_state")
        N = q.mesh.ndof
        # columns of A as rows of the tensor (A is column-major)
        return {"At": torch.as_tensor(_DeviceArray(A.value, (N, N), (8 * lda.value, 8), q), device="cuda"),
                "FI": torch.as_tensor(_DeviceArray(FI.value, (N,), (8,), q), device="cuda")}
    if kind == "points":
        q = st["q"]
        if case["host"]:
            u, s, pr, vm = q.compute_internal_points()
            return {"u": u.T, "s": s.T, "pr": pr.T, "vm": vm[:, None]}
        i, o = st["in"], st["out"]
        q.ctx.check(q.ctx.L.bem_internal_points_device(q.ctx.h, q.mesh.l, *(v.data_ptr() for v in i + o), 0),
                    "internal_points_device")
        return dict(zip(("u", "s", "pr", "vm"), o))
    if kind == "batch":
        b = st["batch"].b
        b.assemble()
        b.solve(case["precision"])
        return {"x": np.concatenate([b.solution(i).ravel(order="F") for i in range(case["count"])])}
    if kind == "adjoint":
        m = st["mesh"]
        J, gX, gmu, gnu = adjoint.compliance_gradient(m, range(m.ne // 2, m.ne), q=st["q"])
        return {"J": J, "gX": gX, "gmu": gmu, "gnu": gnu}
    if case["how"] == "dgesv":
        LU, ipiv, X, info = dgesv(st["A"], st["B"], ctx=st["ctx"])
        return {"LU": LU, "ipiv": ipiv, "X": X, "info": info}
    x, _ = solve_system(st["A"], st["B"][:, 0], case["how"], ctx=st["ctx"])
    return {"x": x}


# ----------------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------------

# FP64 operations of one collocation node against one Gauss point: the T* kernel (about
# 60) and its nine components on nine shape functions; of one internal point against one
# Gauss point: displacement and stress identities
_PAIR, _POINT = 60 + 2 * 81, 190


def _asm_work(n, ne):
    return 8.0 * (3 * n) ** 2, float(_PAIR) * 36 * n * ne


def work(case):
    kind = case["kind"]
    if kind == "dense":
        n, r = case["n"], case["nrhs"]
        return {"bytes": 8.0 * (2 * n * n + 2 * n * r), "flops": 2.0 / 3.0 * n ** 3 + 2.0 * n * n * r}
    if kind == "batch":
        by = fl = 0.0
        for i in range(case["count"]):
            k = i % 6 + 1
            ne = 6 * k * k
            n = 4 * ne + 2
            a, f = _asm_work(n, ne)
            by += a + 8.0 * 2 * 3 * n * 8
            fl += f + 2.0 / 3.0 * (3 * n) ** 3 + 16.0 * (3 * n) ** 2
        return {"bytes": by, "flops": fl}
    if kind == "adjoint":
        ne = 12 * case["m"] ** 2
        n = 4 * ne + 4
        a, f = _asm_work(n, ne)  # the backward assembly visits every pair once more
        return {"bytes": a, "flops": 2 * f + 2.0 / 3.0 * (3.0 * n) ** 3}
    kx, ky, kz = case["kx"], case["ky"], case["kz"]
    ne = 2 * (kx * ky + ky * kz + kz * kx)
    n = 4 * ne + 2
    N = 3.0 * n
    a, f = _asm_work(n, ne)
    pts = (13 * 8.0 * case.get("points", 0), float(_POINT) * 36 * ne * case.get("points", 0))
    if kind == "assembly":
        return {"bytes": a, "flops": f}
    if kind == "points":
        return {"bytes": pts[0], "flops": pts[1]}
    return {"bytes": a + pts[0], "flops": f + 2.0 / 3.0 * N ** 3 + pts[1]}


# ----------------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ----------------------------------------------------------------------------------

_XI = ((-1, -1), (0, -1), (1, -1), (1, 0), (1, 1), (0, 1), (-1, 1), (-1, 0), (0, 0))


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(v):
    return torch.as_tensor(np.array(v), device=_dev())


def _shape(g):
    """Quad9 shape functions and derivatives at points g (P, 2), nodes numbered around the
    element: (3, P, 9)."""
    def lag(x):
        v = {-1: 0.5 * x * (x - 1), 0: 1 - x * x, 1: 0.5 * x * (x + 1)}
        return v, {-1: x - 0.5, 0: -2 * x, 1: x + 0.5}
    (a, da), (b, db) = lag(g[:, 0]), lag(g[:, 1])
    return torch.stack([torch.stack([p[i] * q[j] for i, j in _XI], -1) for p, q in ((a, b), (da, b), (a, db))])


@functools.lru_cache(maxsize=None)
def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    g = np.stack(np.meshgrid(x, x, indexing="ij"), -1).reshape(-1, 2)
    return _t(g), _t(np.outer(w, w).reshape(-1))


@functools.lru_cache(maxsize=None)
def _singular(k):
    """Points and weights of the element seen from its node k: 6 x 6 rules on the triangles
    that the node forms with the corner-to-corner sides it does not lie on."""
    x, w = np.polynomial.legendre.leggauss(6)
    v, corner = np.array(_XI[k], float), np.array([_XI[0], _XI[2], _XI[4], _XI[6]], float)
    g, wt = [], []
    for s in range(4):
        a, b = corner[s] - v, corner[(s + 1) % 4] - v
        area = 0.5 * (a[0] * b[1] - a[1] * b[0])
        if area < 1e-12:
            continue
        s1, s2 = (m.reshape(-1, 1) for m in np.meshgrid(0.5 * (x + 1), 0.5 * (x + 1), indexing="ij"))
        g.append(v + s1 * ((1 - s2) * a + s2 * b))
        wt.append((2 * area * s1[:, 0]) * 0.25 * np.outer(w, w).reshape(-1))
    return _t(np.concatenate(g)), _t(np.concatenate(wt))


def _surface(Xe, g):
    """Points, unit normals and Jacobians of elements Xe (E, 9, 3) at g: (E, P, ...)."""
    f, d1, d2 = _shape(g)
    cr = torch.cross(d1 @ Xe, d2 @ Xe, dim=-1)
    J = torch.linalg.norm(cr, dim=-1)
    return f, f @ Xe, cr / J[..., None], J


def _kelvin(r, n, mu, nu):
    """U* and T* (..., row, column) for r and n (..., 3)."""
    d2 = (r * r).sum(-1)[..., None, None]
    d = torch.sqrt(d2)
    a = r / d[..., 0]
    an = (a * n).sum(-1)[..., None, None]
    I = torch.eye(3, dtype=r.dtype, device=r.device)  # noqa: E741
    aa = a[..., :, None] * a[..., None, :]
    na = n[..., :, None] * a[..., None, :]
    U = ((3 - 4 * nu) * I + aa) / (16 * math.pi * (1 - nu) * mu * d)
    T = -(an * ((1 - 2 * nu) * I + 3 * aa) + (1 - 2 * nu) * (na - na.mT)) / (8 * math.pi * (1 - nu) * d2)
    return U, T


def _blocks(X, mu, nu, kc, i0, i1):
    """h and g of collocation nodes [i0, i1) against every element: (B, ne, 9, 3, 3), the
    h of a node on itself left zero."""
    ne = kc.shape[0]
    g, w = _gauss(6)
    f, xg, nr, J = _surface(X[kc], g)
    p = f * (J * w)[..., None]  # (ne, 36, 9)
    U, T = _kelvin(xg - X[i0:i1, None, None, :], nr, mu, nu)
    on = (kc[None] == torch.arange(i0, i1, device=kc.device)[:, None, None]).any(-1)
    out = []
    for K in (T, U):
        v = torch.einsum("beqc,eqk->bekc", K.flatten(-2), p).unflatten(-1, (3, 3))
        out.append(torch.where(on[:, :, None, None, None], torch.zeros_like(v), v))
    for k in range(9):  # elements whose node k is one of the rows
        e = ((kc[:, k] >= i0) & (kc[:, k] < i1)).nonzero()[:, 0]
        if not len(e):
            continue
        g, w = _singular(k)
        f, xg, nr, J = _surface(X[kc[e]], g)
        i = kc[e, k]
        U, T = _kelvin(xg - X[i][:, None, :], nr, mu, nu)
        p = f * (J * w)[..., None]
        keep = torch.ones(9, dtype=X.dtype, device=X.device)
        keep[k] = 0.0
        for m, K in enumerate((T, U)):
            v = torch.einsum("eqc,eqk->ekc", K.flatten(-2), p).unflatten(-1, (3, 3))
            out[m] = out[m].index_put((i - i0, e), v * keep[:, None, None] if m == 0 else v, accumulate=True)
    return out


class _Problem:
    """A quad9 mesh's supports and loads as tensors; bc (ne, 9, 3) may carry load cases last."""

    def __init__(self, mesh, bcs=None):
        self.n, self.ne = mesh.n, mesh.ne
        self.X = _t(mesh.node_coords())
        self.kc = _t(mesh.kconec.T.astype(np.int64) - 1)
        self.mu, self.nu = float(mesh.mu), float(mesh.nu)
        self.fixed = _t(mesh.kode.reshape(self.ne, 3) == 0)
        bcs = [mesh.bc] if bcs is None else bcs
        self.bc = torch.stack([_t(b.T.reshape(self.ne, 9, 3)) for b in bcs], -1)
        self.pins = _t(np.array(mesh.pins, dtype=np.int64))
        self.ucol = torch.zeros(self.n, 3, dtype=torch.bool, device=self.X.device)
        self.uval = torch.zeros(self.n, 3, self.bc.shape[-1], dtype=torch.float64, device=self.X.device)
        for e in self.fixed.any(1).nonzero()[:, 0].tolist():
            for c in self.fixed[e].nonzero()[:, 0].tolist():
                self.ucol[self.kc[e], c] = True
                self.uval[self.kc[e], c] = self.bc[e, :, c]

    def _step(self):
        return max(1, min(self.n, 30_000 // self.ne))

    def system(self):
        n, ne, N = self.n, self.ne, 3 * self.n
        A = torch.empty(N, N, dtype=torch.float64, device=self.X.device)
        F = torch.empty(N, self.bc.shape[-1], dtype=torch.float64, device=self.X.device)
        cols = (3 * self.kc[:, :, None] + torch.arange(3, device=self.kc.device)).reshape(-1)
        fix = self.fixed[:, None, :].expand(ne, 9, 3).reshape(-1)
        uc, uv = self.ucol.reshape(-1), self.uval.reshape(N, -1)
        t = torch.where(fix[:, None], torch.zeros_like(self.bc.reshape(27 * ne, -1)), self.bc.reshape(27 * ne, -1))
        for i0 in range(0, n, self._step()):
            i1 = min(n, i0 + self._step())
            h, g = (v.permute(0, 3, 1, 2, 4).reshape(3 * (i1 - i0), 27 * ne)
                    for v in _blocks(self.X, self.mu, self.nu, self.kc, i0, i1))
            H = torch.zeros(3 * (i1 - i0), N, dtype=torch.float64, device=h.device).index_add_(1, cols, h)
            rigid = H.reshape(-1, n, 3).sum(1).reshape(i1 - i0, 3, 3)
            for i in range(i1 - i0):
                H[3 * i: 3 * i + 3, 3 * (i0 + i): 3 * (i0 + i) + 3] -= rigid[i]
            F[3 * i0: 3 * i1] = g @ t - H[:, uc] @ uv[uc]
            H[:, uc] = 0.0
            H.index_add_(1, cols[fix], g[:, fix], alpha=-self.mu)
            A[3 * i0: 3 * i1] = H
        A[self.pins] = 0.0
        A[self.pins, self.pins] = 1.0
        F[self.pins] = 0.0
        return A, F

    def solve(self):
        A, F = self.system()
        x = torch.linalg.solve(A, F)
        return A, x

    def split(self, x):
        """u (n, 3) and t (ne, 9, 3) of the first load case's solution x (3n)."""
        x = x.reshape(self.n, 3)
        u = torch.where(self.ucol, self.uval[..., 0], x)
        return u, torch.where(self.fixed[:, None, :], self.mu * x[self.kc], self.bc[..., 0])


def _principal(s):
    """Principal stresses (descending) and von Mises of s (P, 6) in xx yy zz xy yz zx."""
    S = s[:, [0, 3, 5, 3, 1, 4, 5, 4, 2]].reshape(-1, 3, 3)
    pr = torch.linalg.eigvalsh(S.cpu()).flip(-1).to(s.device)
    d = s[:, :3] - s[:, [1, 2, 0]]
    return pr, torch.sqrt(0.5 * (d * d).sum(1) + 3.0 * (s[:, 3:] ** 2).sum(1))


def _edge_stress(P, u, t):
    """Stresses at the element nodes from in-plane strains and tractions, their nodal means."""
    f, d1, d2 = _shape(_t(np.array(_XI, float)))
    Xe = P.X[P.kc]
    g1, g2 = d1 @ Xe, d2 @ Xe
    e3 = torch.nn.functional.normalize(torch.cross(g1, g2, dim=-1), dim=-1)
    e1 = torch.nn.functional.normalize(g1, dim=-1)
    e2 = torch.cross(e3, e1, dim=-1)
    L = torch.stack([e1, e2, e3], -2)  # (ne, 9, 3, 3)
    # intrinsic derivatives to derivatives along e1 and e2
    M = torch.stack([torch.stack([(g1 * e1).sum(-1), (g1 * e2).sum(-1)], -1),
                     torch.stack([(g2 * e1).sum(-1), (g2 * e2).sum(-1)], -1)], -2)
    du = torch.linalg.solve(M, torch.stack([d1 @ u[P.kc], d2 @ u[P.kc]], -2)) @ L.mT  # [direction, component]
    tl = (L @ t[..., None])[..., 0]
    c = 2 * P.mu / (1 - P.nu)
    k = P.nu / (1 - P.nu)
    S = torch.zeros_like(L)
    S[..., 0, 0] = c * (du[..., 0, 0] + P.nu * du[..., 1, 1]) + k * tl[..., 2]
    S[..., 1, 1] = c * (du[..., 1, 1] + P.nu * du[..., 0, 0]) + k * tl[..., 2]
    S[..., 0, 1] = S[..., 1, 0] = P.mu * (du[..., 0, 1] + du[..., 1, 0])
    for m in range(3):
        S[..., m, 2] = S[..., 2, m] = tl[..., m]
    S = L.mT @ S @ L
    se = torch.stack([S[..., 0, 0], S[..., 1, 1], S[..., 2, 2], S[..., 0, 1], S[..., 1, 2], S[..., 2, 0]], -1)
    cnt = torch.bincount(P.kc.reshape(-1), minlength=P.n)[:, None]
    sn = torch.zeros(P.n, 6, dtype=se.dtype, device=se.device).index_add_(0, P.kc.reshape(-1), se.reshape(-1, 6)) / cnt
    return se, sn


def _somigliana(P, x, y, n, b, t):
    """Displacement and stress at x (..., 1, 3) summed over points y (..., Q, 3) with normals
    n and weighted displacements b and tractions t; the displacement identity keeps the sign
    of the reference's antisymmetric part (stress_mod.f90:838-843)."""
    mu, nu = P.mu, P.nu
    c6 = 1 - 2 * nu
    r = y - x
    d = torch.linalg.norm(r, dim=-1, keepdim=True)
    a = r / d
    dot = lambda p, q: (p * q).sum(-1, keepdim=True)  # noqa: E731
    an, ab, at, nb = dot(a, n), dot(a, b), dot(a, t), dot(n, b)
    k8 = 1 / (8 * math.pi * (1 - nu))
    u = k8 / (2 * mu) / d * ((3 - 4 * nu) * t + a * at) + \
        k8 / d ** 2 * (an * (c6 * b + 3 * a * ab) + c6 * (nb * a - n * ab))
    i, j = [0, 1, 2, 0, 1, 2], [0, 1, 2, 1, 2, 0]
    dl = torch.tensor([1.0, 1, 1, 0, 0, 0], dtype=torch.float64, device=r.device)
    sym = lambda p, q: p[..., i] * q[..., j] + p[..., j] * q[..., i]  # noqa: E731
    aa = a[..., i] * a[..., j]
    D = k8 / d ** 2 * (c6 * (sym(t, a) - dl * at) + 3 * aa * at)
    S = 2 * mu * k8 / d ** 3 * (3 * an * (dl * c6 * ab + nu * sym(b, a) - 5 * aa * ab) + 3 * nu * ab * sym(n, a) +
                                c6 * (3 * nb * aa + sym(n, b)) - (1 - 4 * nu) * nb * dl)
    return u.sum(-2), (D - S).sum(-2)


def _interior(P, u, t, pts):
    pts = _t(pts)
    Xe = P.X[P.kc]
    c = Xe.mean(1)
    lim = 3.5 ** 2 * ((Xe - c[:, None]) ** 2).sum(-1).amax(1)
    tab = []
    for m in (6, 40):
        g, w = _gauss(m)
        f, xg, nr, J = _surface(Xe, g)
        w = (J * w)[..., None]
        tab.append((xg, nr, (f @ u[P.kc]) * w, (f @ t) * w))
    uo = torch.zeros(len(pts), 3, dtype=torch.float64, device=pts.device)
    so = torch.zeros(len(pts), 6, dtype=torch.float64, device=pts.device)
    near = torch.cat([((pts[i: i + 4096, None] - c) ** 2).sum(-1) <= lim for i in range(0, len(pts), 4096)])
    for want, T, per in ((False, tab[0], 36), (True, tab[1], 1600)):
        idx = (near == want).nonzero()
        for k in range(0, len(idx), 4_000_000 // per):
            p, e = idx[k: k + 4_000_000 // per].T
            du, ds = _somigliana(P, pts[p][:, None], *(v[e] for v in T))
            uo.index_add_(0, p, du)
            so.index_add_(0, p, ds)
    return (uo, so) + _principal(so)


def _points_of(mesh):
    return np.stack([mesh.cx, mesh.cy, mesh.cz], 1)


def _host(v):
    return v.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "dense":
        A, B = _dense(case, seed)
        if case["how"] != "dgesv":
            return {"x": np.linalg.solve(A, B[:, 0])}
        LU, _ = torch.linalg.lu_factor(torch.from_numpy(np.ascontiguousarray(A.T)))  # the factors are A^T's
        return {"LU": LU.T.numpy(), "ipiv": None, "X": np.linalg.solve(A, B), "info": None}
    if kind == "batch":
        xs = [_host(_Problem(m, bcs).solve()[1].T.reshape(-1)) for m, bcs in _boxes(case, seed)]
        return {"x": np.concatenate(xs)}
    if kind == "adjoint":
        return _exact_adjoint(_sphere(case, seed))
    mesh = _box(case, seed)
    if mesh.ndof > 20_000:
        return None
    P = _Problem(mesh)
    if kind == "assembly":
        A, F = P.system()
        return {"At": A.T, "FI": F[:, 0]}
    A, x = P.solve()
    x = x[:, 0]
    del A
    u, t = P.split(x)
    if kind == "points":
        return dict(zip(("u", "s", "pr", "vm"), (v.reshape(mesh.l, -1) for v in _interior(P, u, t, _points_of(mesh)))))
    out = {"x": x, "u": u.reshape(-1), "t": t.reshape(P.ne, 27).T}
    if kind == "run":
        se, sn = _edge_stress(P, u, t)
        pr, vm = _principal(sn)
        out.update(sigma_elem=se.permute(2, 1, 0), sigma_node=sn.T, sigma_node_prin=pr.T, sigma_node_vm=vm)
        ui, si, pr, vm = _interior(P, u, t, _points_of(mesh))
        out.update(u_int=ui.T, sigma=si.T, prin=pr.T, vm=vm)
    return {k: _host(v) for k, v in out.items()}


def _exact_adjoint(mesh):
    """J and its gradients: the adjoint identity with the rows of R = lambda^T (FI - A x)
    differentiated by autograd, a few collocation nodes at a time."""
    P = _Problem(mesh)
    A, x = P.solve()
    X, xv = P.X.clone().requires_grad_(), x[:, 0].clone().requires_grad_()
    mu, nu = (torch.tensor(v, dtype=torch.float64, device=X.device, requires_grad=True) for v in (P.mu, P.nu))

    def split(xv):
        x3 = xv.reshape(P.n, 3)
        return (torch.where(P.ucol, P.uval[..., 0], x3),
                torch.where(P.fixed[:, None, :], mu * x3[P.kc], P.bc[..., 0]))

    el = torch.arange(P.ne // 2, P.ne, device=X.device)
    g, w = _gauss(6)
    u, t = split(xv)
    f, _, _, Jac = _surface(X[P.kc[el]], g)
    J = (((f @ u[P.kc[el]]) * (f @ t[el])).sum(-1) * Jac * w).sum()
    J.backward()
    lam = torch.linalg.solve(A.T, xv.grad)
    lam[P.pins] = 0.0
    lam = lam.reshape(P.n, 3)
    del A
    step = max(1, 8_000 // P.ne)
    for i0 in range(0, P.n, step):
        i1 = min(P.n, i0 + step)
        u, t = split(xv.detach())
        h, g = _blocks(X, mu, nu, P.kc, i0, i1)
        rel = u[P.kc][None] - u[i0:i1, None, None, :]  # the rigid-body diagonal
        row = torch.einsum("bekij,ekj->bi", g, t) - torch.einsum("bekij,bekj->bi", h, rel)
        (row * lam[i0:i1]).sum().backward()
    return {"J": float(J.detach()), "gX": _host(X.grad), "gmu": float(mu.grad), "gnu": float(nu.grad)}
