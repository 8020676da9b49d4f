"""The FP64 operator as assembled node rows (csrc/kernels_rows.cuh) against the
FP64 oracle: meshes whose node count falls on, before and after a slice (16
rows) or a window (512 rows), a node with more neighbours than a list sorted by
insertion, partly constrained nodes, per-element moduli.

Tolerances: a row sums at most a few hundred products, each rounded relative to
|K_ij| |x_j - x_i|, and K_ij is a sum over the elements of one edge: 1e-13 of
the result's norm leaves two orders of magnitude.
"""
import numpy as np
import pytest

import oracle as O
from conftest import rel
from cudafemproject_gb300 import meshgen
from cudafemproject_gb300.meshio import Problem

pytestmark = pytest.mark.gpu


def _problem(dim, nodes, elems, cons, young=None):
    z = np.zeros((0, dim))
    return Problem(dim=dim, nodes=np.asarray(nodes, np.float32).astype(np.float64), elems=np.asarray(elems, np.int32),
                   cons=np.asarray(cons, np.int32).reshape(-1, 2), load_node=np.zeros(0, np.int32), load_vec=z,
                   face_nodes=np.zeros((0, dim + 1), np.int32), face_elem=np.zeros(0, np.int32), face_normal=z,
                   face_pressure=np.zeros(0), E=2e7, nu=0.25, rho=2000.0, elem_E=young)


def _strip(n_nodes):
    """A strip of triangles with exactly n_nodes nodes."""
    i = np.arange(n_nodes)
    nodes = np.stack([0.5 * i, (i % 2) * 0.8 + 0.01 * np.sin(i)], axis=1)
    return _problem(2, nodes, np.stack([i[:-2], i[1:-1], i[2:]], axis=1), [[0, 3], [1, 1], [n_nodes - 1, 2]])


def _hub(n_rim):
    """A double cone of tetrahedra around one axis: two nodes with n_rim + 1 neighbours."""
    t = 2 * np.pi * np.arange(n_rim) / n_rim
    nodes = np.concatenate([[[0, 0, -1], [0, 0, 1]], np.stack([np.cos(t), np.sin(t), 0.1 * np.cos(3 * t)], axis=1)])
    i = np.arange(n_rim)
    elems = np.stack([np.zeros_like(i), np.ones_like(i), 2 + i, 2 + (i + 1) % n_rim], axis=1)
    return _problem(3, nodes, elems, [[2, 7], [5, 1], [9, 2]], 2e7 * (1 + 0.5 * np.sin(i)))


MESHES = {
    "tet": lambda: _problem(3, [[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]], [[0, 1, 2, 3]], [[0, 7], [1, 2]]),
    "strip15": lambda: _strip(15),
    "strip16": lambda: _strip(16),
    "strip17": lambda: _strip(17),
    "strip511": lambda: _strip(511),
    "strip512": lambda: _strip(512),
    "strip513": lambda: _strip(513),
    "hub20": lambda: _hub(20),
    "hub300": lambda: _hub(300),
    "delaunay": lambda: meshgen.random_tets(900, seed=11),
    "box_code1": lambda: meshgen.box_3d(5, 4, 11, jitter=0.2, seed=1, clamp_code=1),
    "box_code2": lambda: meshgen.box_3d(5, 4, 11, jitter=0.2, seed=1, clamp_code=2),
}


@pytest.mark.parametrize("name", MESHES)
def test_fp64_rows_against_the_oracle(name):
    from cudafemproject_gb300.solver import FemContext
    p = MESHES[name]()
    ctx, o = FemContext(p), O.Oracle(p)
    x = np.random.default_rng(3).standard_normal(p.n_dof)
    y, ref = ctx.matvec(x, "fp64"), o.matvec(x)
    assert np.linalg.norm(y - ref) <= 1e-13 * np.linalg.norm(ref)
    # values at constrained DOFs reach their own rows only, whatever they are
    bc = ctx.bc_mask().astype(bool)
    free = ~bc
    for bad in (1e200, np.inf, np.nan):
        xb = x.copy()
        xb[bc] = bad
        assert np.array_equal(ctx.matvec(xb, "fp64")[free], y[free])
    # moduli changed in place: the rows are assembled again
    young = 2e7 * np.exp(0.3 * np.random.default_rng(4).standard_normal(p.n_elems))
    ctx.set_young(young)
    p.elem_E = young
    assert rel(ctx.matvec(x, "fp64"), O.Oracle(p).matvec(x)) <= 1e-13


@pytest.mark.parametrize("n", [7, 98, 99, 196, 198])
def test_fp64_pcg_shapes_against_the_oracle(n):
    """The one-kernel PCG in its three shapes (four slices per CTA, one per warp,
    many per warp; 98/99 and 196/198 quads a side lie on either side of the
    limits of a 152-SM GPU): the first two iterates (two recurrences that differ
    in the order of their sums: 1e-12) and the converged solution (1e-10, the
    bar of every FP64 solve)."""
    from cudafemproject_gb300.solver import FemContext
    p = meshgen.square_2d(n)
    f = np.zeros((p.n_nodes, 2))
    f[p.nodes[:, 0] > 1 - 1e-9] = (0.7, -0.2)
    f = f.ravel()
    ctx, o = FemContext(p), O.Oracle(p)
    for iters in (1, 2):
        x, it = o.pcg(f, tol=1e-30, rule=1, maxit=iters, allow_maxit=True)
        u, info = ctx.pcg(f, "fp64", tol=1e-30, stop_rule="residual", max_iter=iters, allow_not_converged=True)
        assert info["iterations"] == it == iters
        assert rel(u, x) <= 1e-12
    u, _ = ctx.pcg(f, "fp64", tol=1e-13, stop_rule="residual")
    assert rel(u, o.pcg(f, tol=1e-13, rule=1)[0]) <= 1e-10


def _column(nx, ny, nz):
    return meshgen.box_3d(nx, ny, nz, lz=4.0, jitter=0.2, seed=5, rho=2000.0, traction=None,
                          point_load=("top_centre", (0.4, -0.3, -1.0)))


@pytest.mark.parametrize("semantics", ["consistent", "compat"])
@pytest.mark.parametrize("mesh,steps", [("tet", 1), ("tet", 2), ("hub300", 5), ("strip513", 6), ("column", 7), ("plate198", 3)])
def test_fp64_explicit_steps_against_the_oracle(semantics, mesh, steps):
    """One-kernel explicit steps, rows in registers (the small meshes) and in
    memory (39,601 nodes: more slices than warps), constant and re-sorted lumped
    masses (segments longer than a staging tile: the hub's 301 elements). The
    recurrence is the oracle's with other summation orders: a few steps stay
    within 1e-11."""
    from cudafemproject_gb300.solver import FemContext
    p = {"column": lambda: _column(4, 3, 17), "plate198": lambda: meshgen.square_2d(198)}.get(mesh, MESHES.get(mesh))()
    if not len(p.face_elem) and not len(p.load_node):
        p.load_node, p.load_vec = np.array([p.n_nodes - 1], np.int32), np.full((1, p.dim), 0.5)
    dt, T = 1e-6, steps * 1e-6 * 1.0000001
    rec = np.array([p.n_nodes - 1, 0, p.n_nodes // 2, p.n_nodes - 1], np.int32)
    ug, st, _ = O.Oracle(p, consistent=semantics == "consistent").dyn(0.5, 0.0, dt, T)
    u, info, trace = FemContext(p, semantics=semantics).dyn(0.5, 0.0, dt, T, precision="fp64", receivers=rec)
    assert info["steps"] == st == steps
    assert rel(u, ug) <= 1e-11
    assert np.array_equal(trace[-1], u[rec])


@pytest.mark.parametrize("states_mb", [None, "0"])
@pytest.mark.parametrize("mesh,steps", [("column", 1), ("column", 16), ("column", 17), ("strip513", 9)])
def test_dyn_adjoint_whole_and_by_segments(monkeypatch, states_mb, mesh, steps):
    """The reverse sweep with every state held and with checkpoints (one segment,
    full ones, a short last one), a receiver listed twice."""
    from cudafemproject_gb300.solver import FemContext
    if states_mb is None:
        monkeypatch.delenv("CFEM_DYN_STATES_MB", raising=False)
    else:
        monkeypatch.setenv("CFEM_DYN_STATES_MB", states_mb)
    p = _column(4, 3, 17) if mesh == "column" else _strip(513)
    if not len(p.load_node):
        p.load_node, p.load_vec = np.array([400], np.int32), np.full((1, 2), 0.5)
    dt, T = 1e-5, steps * 1e-5 * 1.0000001
    rec = np.array([p.n_nodes - 3, p.n_nodes // 2, p.n_nodes - 3], np.int32)
    obs = 1e-9 * np.random.default_rng(1).standard_normal((steps, 3, p.dim))
    L, g, info = FemContext(p, semantics="consistent").dyn_adjoint(0.5, dt, T, rec, obs)
    Lo, go = O.Oracle(p, consistent=True).dyn_adjoint(0.5, dt, T, rec, obs)
    assert info["steps"] == steps
    assert abs(L - Lo) <= 1e-11 * abs(Lo)
    assert rel(g, go) <= 1e-11


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_matvec_on_device_arrays(precision):
    """Device arrays in place, overlapping (x is y), offset to odd elements, and
    host arrays: the same product."""
    import torch
    from cudafemproject_gb300.solver import FemContext
    p = MESHES["box_code1"]()
    ctx = FemContext(p)
    dt, tol = (torch.float64, 0.0) if precision == "fp64" else (torch.float32, 2e-6)
    x = torch.tensor(np.random.default_rng(6).standard_normal(p.n_dof), dtype=dt)
    ref = np.array(ctx.matvec(x.numpy().copy(), precision))
    same = lambda y: np.linalg.norm(y.cpu().numpy() - ref) <= tol * np.linalg.norm(ref)  # FP32 sums are atomic
    xd = x.cuda()
    assert same(ctx.matvec(xd, precision))
    buf = torch.zeros(2 * p.n_dof + 3, dtype=dt, device="cuda")
    xo, yo = buf[1:1 + p.n_dof], buf[2 + p.n_dof:2 + 2 * p.n_dof]
    xo.copy_(xd)
    torch.cuda.synchronize()
    assert same(ctx.matvec(xo, precision, out=yo))
    assert torch.equal(xo, xd) and float(buf[0]) == 0.0 == float(buf[1 + p.n_dof])
    assert same(ctx.matvec(xd, precision, out=xd))


def test_set_young_on_device_and_refused_values():
    """Moduli from a device array equal those from the host; a value that is not
    positive is refused and leaves the operator as it was; the captured FP32
    iterations follow the new moduli."""
    import torch
    from cudafemproject_gb300 import capi
    from cudafemproject_gb300.solver import FemContext
    p = meshgen.box_3d(5, 4, 11, jitter=0.2, seed=1)
    young = 2e7 * np.exp(0.3 * np.random.default_rng(4).standard_normal(p.n_elems))
    f = np.random.default_rng(5).standard_normal(p.n_dof)
    kw = dict(precision="fp32_refine", tol=1e-3, stop_rule="residual", outer_tol=1e-10)
    for form in ("auto", "geometry", "gradient"):
        a, b = FemContext(p, matvec_form=form), FemContext(p, matvec_form=form)
        a.pcg(f, **kw)
        a.set_young(torch.tensor(young, device="cuda"))
        b.set_young(young)
        y = a.matvec(f, "fp64")
        assert np.array_equal(y, b.matvec(f, "fp64"))
        for bad in (0.0, -1.0, np.nan):
            wrong = young.copy()
            wrong[-1] = bad
            with pytest.raises(capi.CfemError):
                a.set_young(wrong)
            assert np.array_equal(a.matvec(f, "fp64"), y)
        p2 = meshgen.box_3d(5, 4, 11, jitter=0.2, seed=1)
        p2.elem_E = young
        assert rel(a.pcg(f, **kw)[0], O.Oracle(p2).pcg(f, tol=1e-13, rule=1)[0]) <= 1e-8


@pytest.mark.parametrize("host_loop", [False, True])
@pytest.mark.parametrize("k", [2, 3, 33, 130])
def test_multi_rhs_case_counts(monkeypatch, host_loop, k):
    """Per-case sums, stopping and FP64 residuals for case counts that fill part of
    a warp, one, several; a case without load, one 1e6 times the others; the
    graph loop and the host loop. Every case within 1e-8 of the oracle."""
    from cudafemproject_gb300.solver import FemContext
    if host_loop:
        monkeypatch.setenv("CFEM_HOST_LOOP", "1")
    else:
        monkeypatch.delenv("CFEM_HOST_LOOP", raising=False)
    p = meshgen.box_3d(4, 3, 9, jitter=0.2, seed=2)
    o = O.Oracle(p, consistent=True).assemble()
    rng = np.random.default_rng(k)
    basis = rng.standard_normal((3, p.n_dof))
    X = np.stack([o.pcg(b, tol=1e-13, rule=1)[0] for b in basis])
    w = rng.standard_normal((k, 3))
    w[1] = 0.0
    w[0] *= 1e6
    ctx = FemContext(p, semantics="consistent")
    for tol in (0.3, 1e-4):
        U, infos = ctx.pcg_multi(w @ basis, precision="fp32_refine", tol=tol, stop_rule="residual", outer_tol=1e-10)
        assert all(i["status"] == 0 for i in infos)
        assert not U[1].any()
        assert max(rel(U[i], w[i] @ X) for i in range(k) if i != 1) <= 1e-8


@pytest.mark.parametrize("live", [(0,), (1, 4), (-1,), (0, 3, -1)])
@pytest.mark.parametrize("width,k", [(2, 32), (4, 64), (8, 64)])
def test_multi_rhs_chunks_that_stop_early(monkeypatch, width, k, live):
    """Several items per CTA (32 or more patches), load in some chunks of `width`
    cases only: the others stop at once and their items are skipped, also where a
    CTA starts and where its range crosses into the next patch. Every case within
    1e-8 of the oracle, the cases without load exactly zero."""
    from cudafemproject_gb300.solver import FemContext
    monkeypatch.setenv("CFEM_MULTI_CASES", str(width))
    p = meshgen.box_3d(6, 5, 17, jitter=0.2, seed=4)
    o = O.Oracle(p, consistent=True).assemble()
    rng = np.random.default_rng(width)
    basis = rng.standard_normal((2, p.n_dof))
    X = np.stack([o.pcg(b, tol=1e-13, rule=1)[0] for b in basis])
    w = np.zeros((k, 2))
    for chunk in live:
        w.reshape(-1, width, 2)[chunk] = rng.standard_normal((width, 2))
    w.reshape(-1, width, 2)[live[0]][1] = 0.0
    ctx = FemContext(p, semantics="consistent", patch_elems=96)
    for tol in (0.3, 1e-4):
        U, infos = ctx.pcg_multi(w @ basis, precision="fp32_refine", tol=tol, stop_rule="residual", outer_tol=1e-10)
        assert all(i["status"] == 0 for i in infos)
        for i in range(k):
            if w[i].any():
                assert rel(U[i], w[i] @ X) <= 1e-8
            else:
                assert not U[i].any()


@pytest.mark.parametrize("rule", ["residual", "reference"])
@pytest.mark.parametrize("tol", [0.2, 0.5])
@pytest.mark.parametrize("k", [2, 9, 33])
def test_multi_rhs_rounds_end_together(k, tol, rule):
    """Loose inner tolerances: cases that reach theirs run on until the round ends,
    the others resume. With a case solved in one iteration (load on constrained
    DOFs only), one without load, and loads of very different size; every case
    within 1e-8 of the oracle. Too few refinement steps, and runs that end at the
    iteration cap: no more steps than asked for, and the case says so."""
    from cudafemproject_gb300.solver import FemContext
    p = meshgen.box_3d(5, 4, 15, jitter=0.2, seed=6)
    o = O.Oracle(p, consistent=True).assemble()
    rng = np.random.default_rng(k)
    basis = rng.standard_normal((3, p.n_dof))
    fixed = np.zeros((p.n_nodes, 3), dtype=bool)
    fixed[p.cons[:, 0]] = True  # (the mesh clamps whole nodes)
    fixed = fixed.ravel()
    assert fixed.any()
    basis[2][~fixed] = 0.0
    X = np.stack([o.pcg(b, tol=1e-13, rule=1)[0] for b in basis])
    w = np.zeros((k, 3))
    w[:, :2] = rng.standard_normal((k, 2)) * 10.0 ** rng.uniform(-3, 3, size=(k, 1))
    w[0] = (0.0, 0.0, 1.0)
    if k > 2:
        w[3] = 0.0
    F = w @ basis
    ctx = FemContext(p, semantics="consistent")
    kw = dict(precision="fp32_refine", tol=tol, stop_rule=rule, outer_tol=1e-10)
    U, infos = ctx.pcg_multi(F, max_outer=400, **kw)
    assert all(i["status"] == 0 and i["rel_residual"] <= 1e-10 for i in infos)
    for i in range(k):
        if w[i].any():
            assert rel(U[i], w[i] @ X) <= 1e-8
        else:
            assert not U[i].any()
    for cap in (100000, 7):
        U, infos = ctx.pcg_multi(F, max_iter=cap, max_outer=2, allow_not_converged=True, **kw)
        assert np.isfinite(U).all() and all(i["outer_iterations"] <= 2 for i in infos)
        assert infos[1]["status"] != 0 and infos[0]["status"] == 0


def test_fp32_implicit_step_that_fails_keeps_the_state_before_it():
    """Steps are queued one ahead: when a step's PCG does not converge, the result is
    the displacement before that step, as when every step is waited for."""
    import ctypes as C
    from cudafemproject_gb300 import capi
    from cudafemproject_gb300.solver import FemContext
    p = _column(4, 3, 17)
    ctx = FemContext(p, semantics="consistent")

    def run(n, tol, cap):
        u = np.zeros(p.n_dof)
        prm = capi.DynParams(0.5, 0.5, 1e-3, n * 1e-3 * 1.0000001, capi.FP32, tol, capi.STOP_RESIDUAL, cap, 1, 0, None, None)
        inf = capi.DynInfo()
        return capi.lib().cfem_dyn(ctx._h, C.byref(prm), None, u.ctypes.data, C.byref(inf)), u, inf.pcg_iterations

    need = []  # iterations of every step
    for n in range(1, 6):
        st, u, its = run(n, 1e-6, 1000)
        assert st == capi.OK
        need.append(its - sum(need))
    cap = need[0]  # the first step just converges; find the first that does not
    first_bad = next((i for i, k in enumerate(need) if k > cap), None)
    if first_bad is None:
        cap, first_bad = max(need) - 1, int(np.argmax(need))
        first_bad = next(i for i, k in enumerate(need) if k > cap)
    st, u, its = run(5, 1e-6, cap)
    assert st == capi.ERR_NOT_CONVERGED
    ref = run(first_bad, 1e-6, 1000)[1] if first_bad else np.zeros(p.n_dof)
    assert np.linalg.norm(u - ref) <= 1e-4 * np.linalg.norm(ref)  # (FP32 sums are atomic)


@pytest.mark.parametrize("semantics", ["consistent", "compat"])
@pytest.mark.parametrize("form", ["auto", "geometry", "gradient"])
@pytest.mark.parametrize("steps", [1, 2, 3, 11, 12, 19])
def test_fp32_explicit_step_counts(semantics, form, steps):
    """FP32 explicit steps: the one-kernel form (stored gradients) and the two-kernel
    forms, fewer steps than one captured cycle, exactly two, a remainder; loads at
    a point and on faces, a wavelet, a receiver trace of every step. The FP32
    recurrence stays within 1e-4 of the FP64 oracle over these few steps (its
    accelerations carry single rounding errors of 6e-8 amplified by cancellation
    at the first arrivals)."""
    from cudafemproject_gb300.meshio import WaveletParams
    from cudafemproject_gb300.solver import FemContext
    p = _column(4, 3, 17) if steps % 2 else meshgen.box_3d(4, 3, 17, jitter=0.2, seed=5, rho=2000.0)
    w = WaveletParams("ricker", 40.0, 0.0, 1.0)
    dt, T = 2e-5, steps * 2e-5 * 1.0000001
    o = O.Oracle(p, consistent=semantics == "consistent")
    ug, st, _ = o.dyn(0.5, 0.0, dt, T, wavelet=w)
    rec = np.array([p.n_nodes - 1, p.n_nodes // 2], np.int32)
    u, info, trace = FemContext(p, semantics=semantics, matvec_form=form).dyn(
        0.5, 0.0, dt, T, precision="fp32", wavelet=w, receivers=rec)
    assert info["steps"] == st == steps
    assert rel(u, ug) <= 1e-4
    _, _, t64 = FemContext(p, semantics=semantics).dyn(0.5, 0.0, dt, T, precision="fp64", wavelet=w, receivers=rec)
    assert np.array_equal(trace[-1], u[rec])
    assert rel(trace, t64) <= 1e-4
