"""The calls whose speed this framework is measured by, with inputs made from a seed.

Every case goes through the public Python entry points (FemContext,
BatchContext, autograd.static_solve) the way a program that owns a mesh uses
them: the context is the plan such a program keeps, loads, moduli and
displacements are what changes from call to call. ``exact`` gives the same
results in 64 bits from plain torch (element matrices assembled into one sparse
matrix, conjugate gradients to the rounding floor, time stepping and its
adjoint written out), without the framework's kernels; the seeded mesh
generators only supply coordinates and connectivity.
"""
import dataclasses
import functools
import math

import numpy as np
import torch

from cudafemproject_gb300 import meshgen
from cudafemproject_gb300.meshio import WaveletParams

E0, NU, RHO = 2e7, 0.25, 2000.0


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # one operator application inside a caller's own Krylov or eigenvalue loop on a small
        # mesh: the smallest call, latency and launches
        dict(name="apply_small_fp64", kind="apply", nx=8, ny=8, nz=32, precision="fp64"),
        # the same on a mesh of 0.4 M DOF in single precision: bandwidth
        dict(name="apply_large_fp32", kind="apply", nx=32, ny=32, nz=128, precision="fp32"),
        # the 2D plane-stress square (8192 triangles): FP64 Jacobi-PCG to 1e-12, then stress recovery
        dict(name="plate_fp64", kind="plate", n=64, precision="fp64", tol=1e-12),
        # the 1.39M-DOF jittered cantilever: FP32 PCG with FP64 refinement, the largest solve
        dict(name="cantilever_refine", kind="solve", mesh="box", nx=48, ny=48, nz=192, precision="fp32_refine", tol=1e-3),
        # an unstructured mesh (Delaunay tetrahedra, ragged fans and node degrees) in plain FP64
        dict(name="unstructured_fp64", kind="solve", mesh="delaunay", points=20000, precision="fp64", tol=1e-8),
        # many load cases on one mesh in one call
        dict(name="multi_rhs", kind="multi", nx=16, ny=16, nz=64, k=32, precision="fp32_refine", tol=0.2),
        # independent meshes of uneven sizes and materials in one call
        dict(name="batch_boxes", kind="batch", boxes=12, n_min=6, n_max=20, precision="fp32_refine", tol=1e-4),
        # one step of a modulus inversion: new per-element moduli, forward solve, adjoint gradient
        dict(name="inversion_step", kind="inversion", nx=16, ny=16, nz=64, precision="fp32_refine", tol=0.4),
        # explicit elastodynamics with a Ricker source and receivers, single precision
        dict(name="explicit_fp32", kind="explicit", semantics="consistent", nx=24, ny=24, nz=192, steps=400, precision="fp32"),
        # the same path with the reference's own semantics and precision (the defaults of a FemContext)
        dict(name="explicit_reference", kind="explicit", semantics="compat", nx=16, ny=16, nz=128, steps=100, precision="fp64"),
        # implicit Newmark steps with consistent mass, warm-started PCG per step
        dict(name="implicit_fp32", kind="implicit", nx=16, ny=16, nz=128, steps=20, precision="fp32", tol=1e-6),
        # receiver-misfit gradient back through explicit time steps
        dict(name="dyn_adjoint", kind="dyn_adjoint", nx=10, ny=10, nz=40, steps=120),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi, stretch=(2.0, 8.0)):
    """Box counts around one size, not equal to each other, odd ones among them."""
    n = _log_int(rng, lo, hi)
    return dict(nx=max(2, n + rng.randint(-1, 2)), ny=max(2, n + rng.randint(-1, 2)),
                nz=int(n * rng.uniform(*stretch)) + 1)


def draw(rng):
    kind = rng.choice(["apply", "plate", "solve", "multi", "batch", "inversion", "explicit", "implicit", "dyn_adjoint"])
    if kind == "apply":
        return dict(kind=kind, **_box(rng, 3, 34, (2.0, 4.0)), precision=rng.choice(["fp64", "fp32"]))
    if kind == "plate":
        return dict(kind=kind, n=_log_int(rng, 8, 180), precision=rng.choice(["fp64", "fp32_refine"]), tol=1e-12)
    if kind == "solve":
        precision = rng.choice(["fp64", "fp32_refine"])
        tol = 1e-8 if precision == "fp64" else rng.choice([0.3, 0.4, 1e-3])
        if rng.random() < 0.4:
            return dict(kind=kind, mesh="delaunay", points=_log_int(rng, 600, 40000), precision=precision, tol=tol)
        return dict(kind=kind, mesh="box", **_box(rng, 4, 20 if precision == "fp64" else 32, (2.0, 4.0)),
                    precision=precision, tol=tol)
    if kind == "multi":
        return dict(kind=kind, **_box(rng, 4, 16, (2.0, 4.0)), k=_log_int(rng, 2, 48), precision="fp32_refine", tol=rng.choice([0.2, 1e-3]))
    if kind == "batch":
        return dict(kind=kind, boxes=_log_int(rng, 2, 16), n_min=4, n_max=_log_int(rng, 6, 20), precision="fp32_refine",
                    tol=rng.choice([0.3, 1e-4]))
    if kind == "inversion":
        return dict(kind=kind, **_box(rng, 4, 18, (2.0, 4.0)), precision=rng.choice(["fp64", "fp32_refine", "fp32_refine"]), tol=0.4)
    if kind == "explicit":
        semantics = rng.choice(["compat", "consistent"])
        return dict(kind=kind, semantics=semantics, **_box(rng, 4, 20 if semantics == "consistent" else 14),
                    steps=_log_int(rng, 20, 400 if semantics == "consistent" else 100), precision=rng.choice(["fp64", "fp32"]))
    if kind == "implicit":
        return dict(kind=kind, **_box(rng, 4, 16), steps=_log_int(rng, 2, 24), precision="fp32", tol=1e-6)
    return dict(kind=kind, **_box(rng, 3, 11, (2.0, 4.0)), steps=_log_int(rng, 20, 150))


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=4)
def _mesh_of(key):
    kind, a, b, c, extra = key
    if kind == "plate":
        return meshgen.square_2d(a, E=E0, nu=NU)
    if kind == "delaunay":
        return meshgen.random_tets(a, seed=7, E=E0, nu=NU, rho=RHO)
    load = None
    if extra in ("explicit", "implicit", "dyn_adjoint"):
        load = ("top_centre", (0.3, 0.2, -1.0))
    lz = 4.0 if extra == "solve" else 8.0
    return meshgen.box_3d(a, b, c, lz=lz, jitter=0.2, seed=0, E=E0, nu=NU, rho=RHO,
                          traction=None if load else (0.0, -1e3, 0.0), point_load=load)


def _mesh(case):
    k = case["kind"]
    if k == "plate":
        return _mesh_of(("plate", case["n"], 0, 0, ""))
    if case.get("mesh") == "delaunay":
        return _mesh_of(("delaunay", case["points"], 0, 0, ""))
    extra = k if k in ("explicit", "implicit", "dyn_adjoint") else "solve"
    return _mesh_of(("box", case["nx"], case["ny"], case["nz"], extra))


def _batch_meshes(case, seed):
    """Boxes n x n x 4n of fixed uneven sizes, materials and loads from the seed."""
    sizes = np.random.default_rng(2).integers(case["n_min"], case["n_max"] + 1, size=case["boxes"])
    rng = np.random.default_rng(seed)
    return [meshgen.box_3d(int(n), int(n), 4 * int(n), jitter=0.2, seed=3 + i, E=float(10.0 ** rng.uniform(6, 8)),
                           nu=float(rng.uniform(0.2, 0.4)), traction=tuple(1e3 * rng.standard_normal(3)))
            for i, n in enumerate(sizes)]


def _constrained(p):
    """[n_dof] bool: clamped DOFs (these meshes clamp whole nodes)."""
    m = np.zeros((p.n_nodes, p.dim), bool)
    m[p.cons[:, 0]] = True
    return m.reshape(-1)


def _loads(p, seed, k=1):
    """[k][n_dof] nodal loads: a force of random direction and magnitude spread
    evenly over the nodes of the free end."""
    rng = np.random.default_rng(seed)
    axis = 0 if p.dim == 2 else 2
    x = p.nodes[:, axis]
    end = x >= x.max() - 1e-9
    if not len(p.face_elem):  # no flat end face: a layer of nodes
        end = x >= x.max() - 0.05 * (x.max() - x.min())
    d = rng.standard_normal((k, p.dim))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    f = np.zeros((k, p.n_nodes, p.dim))
    f[:, end] = (10.0 ** rng.uniform(2, 4, size=(k, 1)) * d / end.sum())[:, None, :]
    return f.reshape(k, -1)


def _young(p, seed):
    return E0 * np.exp(0.5 * np.random.default_rng(seed + 1).standard_normal(p.n_elems))


def _dof_field(p, seed):
    return np.random.default_rng(seed + 2).standard_normal(p.n_dof)


def _dt(case):
    n = max(case["nx"], case["ny"], case["nz"] / 8.0)
    return float(np.float32((4e-4 if case.get("semantics") == "compat" else 1e-3) / n))


def _wave(seed):
    r = np.random.default_rng(seed + 3)
    return WaveletParams("ricker", float(np.float32(r.uniform(20.0, 60.0))), 0.0, 1.0)


def _receivers(p, seed, n=24):
    """The loaded node and others of the free end face, where the waves arrive."""
    x = p.nodes[:, 2]
    end = np.setdiff1d(np.nonzero(x >= x.max() - 1e-9)[0], p.load_node)
    pick = np.random.default_rng(seed + 4).choice(end, size=min(n - 1, len(end)), replace=False)
    return np.sort(np.concatenate([p.load_node, pick])).astype(np.int32)


def _observations(p, case, seed):
    n = len(_receivers(p, seed))
    return 1e-9 * np.random.default_rng(seed + 5).standard_normal((case["steps"], n, 3))


def _endtime(case):
    return case["steps"] * _dt(case) * 1.0000001


def _problem_for_steps(case, seed):
    """The dynamics mesh with this seed's point load at the top centre."""
    p = _mesh(case)
    v = np.random.default_rng(seed + 6).standard_normal((1, 3))
    return dataclasses.replace(p, load_vec=(v / np.linalg.norm(v)).astype(np.float32).astype(np.float64))


def prepare(case, seed):
    from cudafemproject_gb300.solver import BatchContext, FemContext
    kind = case["kind"]
    s = dict(case=dict(case))
    if kind == "batch":
        s["fem"] = BatchContext(_batch_meshes(case, seed))
        return s
    if kind in ("explicit", "implicit", "dyn_adjoint"):
        p = _problem_for_steps(case, seed)
        s["fem"] = FemContext(p, semantics=case.get("semantics", "consistent"))
        s["dt"], s["wave"], s["receivers"] = _dt(case), _wave(seed), _receivers(p, seed)
        if kind == "implicit":
            s["dt"] = 1e-3
        if kind == "dyn_adjoint":
            s["obs"] = _observations(p, case, seed)
        return s
    p = _mesh(case)
    s["fem"] = FemContext(p, semantics="consistent")
    if kind == "apply":
        dt = torch.float64 if case["precision"] == "fp64" else torch.float32
        s["x"] = torch.tensor(_dof_field(p, seed), dtype=dt, device="cuda")
        s["y"] = torch.empty_like(s["x"])
    elif kind == "plate":
        s["f"] = _loads(p, seed)[0]
    elif kind == "solve":
        s["f"] = torch.tensor(_loads(p, seed)[0], device="cuda")
        s["u"] = torch.zeros_like(s["f"])
    elif kind == "multi":
        s["F"] = _loads(p, seed, case["k"])
    elif kind == "inversion":
        s["young"] = torch.tensor(_young(p, seed), device="cuda", requires_grad=True)
        s["f"] = torch.tensor(_loads(p, seed)[0], device="cuda", requires_grad=True)
        s["g"] = torch.tensor(_dof_field(p, seed), device="cuda")
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    c, fem = s["case"], s["fem"]
    kind = c["kind"]
    if kind == "apply":
        return fem.matvec(s["x"], precision=c["precision"], out=s["y"])
    if kind == "plate":
        u, _ = fem.pcg(s["f"], precision=c["precision"], tol=0.4 if c["precision"] != "fp64" else c["tol"],
                       stop_rule="residual", outer_tol=c["tol"])
        strain, stress, mises = fem.element_stress(u)
        return dict(u=u, strain=strain, stress=stress, mises=mises)
    if kind == "solve":
        u, _ = fem.pcg(s["f"], precision=c["precision"], tol=c["tol"], stop_rule="residual", outer_tol=1e-9, out=s["u"])
        return u
    if kind == "multi":
        U, _ = fem.pcg_multi(s["F"], precision=c["precision"], tol=c["tol"], stop_rule="residual", outer_tol=1e-9)
        return U
    if kind == "batch":
        us, _ = fem.static_solve(precision=c["precision"], tol=c["tol"], outer_tol=1e-9)
        return us
    if kind == "inversion":
        from cudafemproject_gb300.autograd import static_solve
        tol = c["tol"] if c["precision"] != "fp64" else 1e-11
        u = static_solve(fem, s["young"], s["f"], precision=c["precision"], tol=tol)
        dE, df = torch.autograd.grad(u, (s["young"], s["f"]), s["g"])
        return dict(u=u.detach(), dE=dE, df=df)
    if kind == "explicit":
        u, _, trace = fem.dyn(0.5, 0.0, s["dt"], _endtime(c), precision=c["precision"],
                              wavelet=s["wave"], receivers=s["receivers"])
        return dict(u=u, trace=trace)
    if kind == "implicit":
        u, _, trace = fem.dyn(0.5, 0.5, s["dt"], c["steps"] * s["dt"] * 1.0000001, precision=c["precision"],
                              wavelet=s["wave"], pcg_tol=c["tol"], stop_rule="residual", receivers=s["receivers"])
        return dict(u=u, trace=trace)
    loss, dE, _ = fem.dyn_adjoint(0.5, s["dt"], _endtime(c), s["receivers"], s["obs"], wavelet=s["wave"])
    return dict(loss=loss, dE=dE)


# ------------------------------------------------------------------ the work of one pass
def _sizes(case):
    """(nodes, elements, values per node) without building the mesh."""
    if case["kind"] == "plate":
        return (case["n"] + 1) ** 2, 2 * case["n"] ** 2, 2
    if case["kind"] == "batch":
        n = 0.5 * (case["n_min"] + case["n_max"])
        return case["boxes"] * 4 * n ** 3, case["boxes"] * 24 * n ** 3, 3
    if case.get("mesh") == "delaunay":
        return case["points"], 5.7 * case["points"], 3
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return (nx + 1) * (ny + 1) * (nz + 1), 6 * nx * ny * nz, 3


def work(case):
    """Inputs once and outputs once; arithmetic of the operator applications
    (gradient form, 150 operations per tetrahedron, 48 per triangle) and vector
    updates, with the iteration counts that Jacobi-PCG needs on these meshes."""
    n, e, dim = _sizes(case)
    kind = case["kind"]
    word = 4 if case.get("precision") in ("fp32", "fp32_refine") else 8
    op = e * (150 if dim == 3 else 48)
    vec = n * dim * 12
    mesh = n * dim * word + e * (dim + 1) * 4
    io = 16 * n * dim
    if kind == "apply":
        return dict(bytes=mesh + 2 * n * dim * word, flops=op)
    if kind == "plate":
        its = 7 * case["n"]
        return dict(bytes=mesh + io + e * 7 * 8, flops=its * (op + vec))
    if kind in ("solve", "inversion"):
        its = 17 * case["nz"] if "nz" in case else 24 * case["points"] ** (1 / 3)
        if kind == "inversion":
            return dict(bytes=mesh + 2 * io + 16 * e, flops=2.4 * its * (op + vec))
        return dict(bytes=mesh + io, flops=its * (op + vec))
    if kind == "multi":
        return dict(bytes=mesh + case["k"] * io, flops=17 * case["nz"] * case["k"] * (op + vec))
    if kind == "batch":
        return dict(bytes=mesh + io, flops=17 * 2 * (case["n_min"] + case["n_max"]) * (op + vec))
    steps = case["steps"]
    out = io + steps * 24 * 3 * 8
    if kind == "explicit":
        return dict(bytes=mesh + out, flops=steps * (op + vec))
    if kind == "implicit":
        return dict(bytes=mesh + out, flops=steps * 20 * (op + vec))
    return dict(bytes=mesh + out + 8 * e, flops=4 * steps * (op + vec))


# ------------------------------------------------------------------ the same in 64 bits
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Operator:
    """Linear elasticity on one mesh in 64 bits: shape gradients per element,
    the constrained stiffness K' = P K P + (I - P) diag(K) as a sparse matrix."""

    def __init__(self, p, young=None):
        dev = _device()
        self.p, self.dim = p, p.dim
        X = torch.tensor(p.nodes, dtype=torch.float64, device=dev)
        self.conn = torch.tensor(p.elems, dtype=torch.int64, device=dev)
        D = p.dim
        J = X[self.conn[:, 1:]] - X[self.conn[:, :1]]
        inv = torch.linalg.inv(J)  # columns: gradients of N_1 .. N_dim
        g = inv.transpose(1, 2)
        self.g = torch.cat([-g.sum(1, keepdim=True), g], 1)
        self.V = torch.linalg.det(J).abs() / (6.0 if D == 3 else 2.0)
        E = torch.full_like(self.V, float(p.E)) if young is None else torch.tensor(young, dtype=torch.float64, device=dev)
        self.E = E
        self.lam1 = p.nu / ((1 + p.nu) * (1 - 2 * p.nu)) if D == 3 else p.nu / (1 - p.nu ** 2)
        self.mu1 = 0.5 / (1 + p.nu)
        self.fixed = torch.tensor(_constrained(p), device=dev)
        self.n = p.n_dof
        self.dofs = (self.conn[:, :, None] * D + torch.arange(D, device=dev)).reshape(len(self.conn), -1)
        self._csr = None

    def energies(self, u, w, E=None):
        """w_e^T K_e u_e of every element over the unconstrained DOFs (K_e with modulus E)."""
        E = self.E if E is None else E
        Hu = torch.einsum("eai,eaj->eij", torch.where(self.fixed, 0.0, u)[self.dofs].view(-1, self.dim + 1, self.dim), self.g)
        Hw = torch.einsum("eai,eaj->eij", torch.where(self.fixed, 0.0, w)[self.dofs].view(-1, self.dim + 1, self.dim), self.g)
        tr = lambda h: h.diagonal(dim1=1, dim2=2).sum(1)
        return self.V * E * (self.lam1 * tr(Hu) * tr(Hw) + self.mu1 * ((Hu + Hu.transpose(1, 2)) * Hw).sum((1, 2)))

    def diagonal(self):
        sq = self.g ** 2
        kd = (self.V * self.E)[:, None, None] * ((self.lam1 + self.mu1) * sq + self.mu1 * sq.sum(2, keepdim=True))
        return torch.zeros(self.n, dtype=torch.float64, device=kd.device).index_add_(0, self.dofs.reshape(-1), kd.reshape(-1))

    def forces(self, x):
        """K' x by elements."""
        u = torch.where(self.fixed, 0.0, x)
        H = torch.einsum("eai,eaj->eij", u[self.dofs].view(-1, self.dim + 1, self.dim), self.g)
        tr = H.diagonal(dim1=1, dim2=2).sum(1)
        eye = torch.eye(self.dim, dtype=torch.float64, device=x.device)
        S = (self.V * self.E)[:, None, None] * (self.lam1 * tr[:, None, None] * eye + self.mu1 * (H + H.transpose(1, 2)))
        f = torch.einsum("eij,eaj->eai", S, self.g)
        y = torch.zeros_like(x).index_add_(0, self.dofs.reshape(-1), f.reshape(-1))
        return torch.where(self.fixed, self.diagonal() * x, y)

    def matrix(self, c_m=0.0, c_k=1.0):
        """c_m M + c_k K (consistent mass) under the constraint mask, as CSR, and its diagonal."""
        D, nv = self.dim, self.dim + 1
        g, eye = self.g, torch.eye(D, dtype=torch.float64, device=self.g.device)
        VE = c_k * self.V * self.E
        dot = torch.einsum("eak,ebk->eab", g, g)
        K = self.lam1 * torch.einsum("eap,ebq->eapbq", g, g) + self.mu1 * torch.einsum("eaq,ebp->eapbq", g, g)
        K += self.mu1 * torch.einsum("eab,pq->eapbq", dot, eye)
        K *= VE[:, None, None, None, None]
        if c_m:
            m = c_m * self.p.rho * self.V / (20.0 if D == 3 else 12.0)
            K += torch.einsum("e,ab,pq->eapbq", m, torch.ones_like(dot[0]) + torch.eye(nv, dtype=torch.float64, device=g.device), eye)
        w = nv * D
        K = K.reshape(-1, w, w)
        fx = self.fixed[self.dofs]
        off = ~torch.eye(w, dtype=torch.bool, device=g.device)
        K.masked_fill_((fx[:, :, None] | fx[:, None, :]) & off, 0.0)
        rows = self.dofs[:, :, None].expand(-1, w, w).reshape(-1)
        cols = self.dofs[:, None, :].expand(-1, w, w).reshape(-1)
        A = torch.sparse_coo_tensor(torch.stack([rows, cols]), K.reshape(-1), (self.n, self.n)).coalesce()
        i, v = A.indices(), A.values()
        on = i[0] == i[1]
        diag = torch.zeros(self.n, dtype=torch.float64, device=g.device).index_add_(0, i[0][on], v[on])
        return A.to_sparse_csr(), diag


def _cg(A, diag, b, x=None, rel=1e-14, cap=60000):
    """Jacobi conjugate gradients to the rounding floor: restarted from the true residual."""
    x = torch.zeros_like(b) if x is None else x.clone()
    nb = b.norm()
    if not float(nb):
        return x
    for _ in range(4):
        r = b - A @ x
        if float(r.norm()) <= rel * float(nb):
            break
        target = max(1e-7 * float(r.norm()), 0.1 * rel * float(nb))
        z = r / diag
        p, gam = z.clone(), r @ z
        for it in range(cap):
            q = A @ p
            a = gam / (p @ q)
            x = x + a * p
            r = r - a * q
            z = r / diag
            new = r @ z
            p = z + (new / gam) * p
            gam = new
            if it % 25 == 24 and float(r.norm()) <= target:
                break
    return x


def _ricker(w, t):
    """The load factor at float time t, in 32-bit arithmetic as the path defines it."""
    tmp = np.float32(math.pi * w.freq * float(t) - math.pi)
    sq = np.float32(tmp * tmp)
    return float(np.float32(np.float32(1) - np.float32(2) * sq) * np.float32(math.exp(-float(sq))))


def _tensor(a):
    return torch.tensor(a, dtype=torch.float64, device=_device())


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        out = []
        for p in _batch_meshes(case, seed):
            op = _Operator(p)
            f = torch.zeros(p.n_nodes, 3, dtype=torch.float64, device=_device())
            fn = torch.tensor(p.face_nodes[:, :3], dtype=torch.int64, device=_device())
            X = _tensor(p.nodes)[fn]
            area = 0.5 * torch.linalg.cross(X[:, 1] - X[:, 0], X[:, 2] - X[:, 0]).norm(dim=1)
            t = _tensor(-p.face_pressure[:, None] * p.face_normal) * (area / 3.0)[:, None]
            for a in range(3):
                f.index_add_(0, fn[:, a], t)
            f = torch.where(op.fixed, 0.0, f.reshape(-1))
            out.append(_cg(*op.matrix(), f).view(-1, 3))
        return out
    if kind in ("explicit", "implicit", "dyn_adjoint"):
        return _exact_steps(case, seed)
    p = _mesh(case)
    if kind == "apply":
        x = torch.tensor(_dof_field(p, seed), dtype=torch.float64 if case["precision"] == "fp64" else torch.float32)
        return _Operator(p).forces(x.double().to(_device()))
    if kind == "inversion":
        op = _Operator(p, _young(p, seed))
        A, d = op.matrix()
        u = _cg(A, d, _tensor(_loads(p, seed)[0]))
        lam = _cg(A, d, _tensor(_dof_field(p, seed)))
        return dict(u=u, dE=-op.energies(u, lam) / op.E, df=lam)
    op = _Operator(p)
    A, d = op.matrix()
    if kind == "multi":
        return torch.stack([_cg(A, d, f) for f in _tensor(_loads(p, seed, case["k"]))]) if case["k"] <= 32 else None
    u = _cg(A, d, _tensor(_loads(p, seed)[0]))
    if kind == "solve":
        return u
    H = torch.einsum("eai,eaj->eij", u[op.dofs].view(-1, 3, 2), op.g)
    strain = torch.stack([H[:, 0, 0], H[:, 1, 1], H[:, 0, 1] + H[:, 1, 0]], 1)
    tr = strain[:, 0] + strain[:, 1]
    stress = op.E[:, None] * torch.stack([op.lam1 * tr + 2 * op.mu1 * strain[:, 0], op.lam1 * tr + 2 * op.mu1 * strain[:, 1],
                                          op.mu1 * strain[:, 2]], 1)
    mises = torch.sqrt(stress[:, 0] ** 2 - stress[:, 0] * stress[:, 1] + stress[:, 1] ** 2 + 3 * stress[:, 2] ** 2)
    return dict(u=u, strain=strain, stress=stress, mises=mises)


def _exact_steps(case, seed):
    """Generalised Newmark steps written out: predictor, acceleration, corrector."""
    p = _problem_for_steps(case, seed)
    op, N, wave = _Operator(p), case["steps"], _wave(seed)
    dt = 1e-3 if case["kind"] == "implicit" else _dt(case)
    compat = case.get("semantics") == "compat"
    f = torch.zeros(p.n_nodes, 3, dtype=torch.float64, device=_device())
    node = int(p.load_node[0])
    # the reference adds a point load once per adjacent element and leaves it constant in time
    f[node] = _tensor(p.load_vec[0]) * (float((p.elems == node).sum()) if compat else 1.0)
    f = f.reshape(-1)
    factor = [1.0 if compat else _ricker(wave, np.float32(np.float32(s) * np.float32(dt))) for s in range(N + 1)]
    rec = torch.tensor(_receivers(p, seed).astype(np.int64), device=_device())
    slots = op.dofs.reshape(-1)
    lump = (p.rho * op.V / (12.0 if compat else 4.0)).repeat_interleave(12)
    # the reference sorts the element masses by DOF in place at every assembly
    perm = torch.argsort(slots, stable=True) if compat else None
    owner = slots[perm] if compat else slots

    def masses(src):
        return torch.zeros(op.n, dtype=torch.float64, device=src.device).index_add_(0, owner, src)

    if case["kind"] == "dyn_adjoint":
        return _exact_adjoint(case, seed, op, f, factor, rec, masses(lump), dt)
    beta2 = 0.5 if case["kind"] == "implicit" else 0.0
    A, _ = op.matrix()
    M = None if compat else masses(lump)
    if beta2:
        Aop, dop = op.matrix(1.0, 0.5 * beta2 * dt * dt)
    d = torch.zeros(op.n, dtype=torch.float64, device=_device())
    v, a, trace = d.clone(), d.clone(), []
    for s in range(1, N + 1):
        d = d + dt * v + 0.5 * (1 - beta2) * dt * dt * a
        r = factor[s] * f - A @ d
        if beta2:
            new = _cg(Aop, dop, r, a)
        else:
            if compat:
                lump = lump[perm]
                M = masses(lump)
            new = r / M
        v = v + 0.5 * dt * (a + new)
        d = d + 0.5 * beta2 * dt * dt * new
        a = new
        trace.append(d.view(-1, 3)[rec])
    return dict(u=d.view(-1, 3), trace=torch.stack(trace))


def _exact_adjoint(case, seed, op, f, factor, rec, M, dt):
    """Loss and modulus gradient of the explicit steps: reverse sweep over the stored trajectory."""
    N, n = case["steps"], op.n
    obs = _tensor(_observations(op.p, case, seed))
    A, _ = op.matrix()
    d = torch.zeros(n, dtype=torch.float64, device=f.device)
    v, a, states, loss = d.clone(), d.clone(), [], 0.0
    miss = []
    for s in range(1, N + 1):
        d = d + dt * v + 0.5 * dt * dt * a
        new = (factor[s] * f - A @ d) / M
        v = v + 0.5 * dt * (a + new)
        a = new
        states.append(d)
        miss.append(d.view(-1, 3)[rec] - obs[s - 1])
        loss = loss + 0.5 * float((miss[-1] ** 2).sum())
    gE = torch.zeros_like(op.E)
    db, vb, ab = torch.zeros_like(d), torch.zeros_like(d), torch.zeros_like(d)
    for s in range(N, 0, -1):
        db.view(-1, 3).index_add_(0, rec, miss[s - 1])
        w = (ab + 0.5 * dt * vb) / M  # adjoint of the acceleration through a = (F - K d) / M
        ab = 0.5 * dt * vb
        gE -= op.energies(states[s - 1], w) / op.E
        db = db - A @ w
        vb = vb + dt * db
        ab = ab + 0.5 * dt * dt * db
    return dict(loss=loss, dE=gE)
