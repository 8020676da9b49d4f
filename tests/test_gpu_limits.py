"""Calls at their limits: loads that underflow in single precision, bodies that
need thousands of iterations, contexts that step in several threads, time steps
that do not converge, iteration caps, little free memory, nodes of many elements,
kernels whose CTAs do not all arrive, traces row by row."""
import numpy as np
import pytest

import oracle as O
from conftest import rel
from cudafemproject_gb300 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rule", ["residual", "reference"])
@pytest.mark.parametrize("tol", [1e-3, 0.1, 0.4])
def test_refinement_of_loads_below_single_precision(tol, rule):
    """Entries of 1e-20: r.z = r^2 / diag(K) is 1e-47, zero in FP32, where r.r =
    1e-40 is not. The FP32 runs take no step, and the solve ends at the second
    step that reduces nothing, with tight inner tolerances as with loose ones. The same load at a size that single precision holds is solved."""
    from cudafemproject_gb300.solver import FemContext
    p = meshgen.box_3d(3, 3, 9, jitter=0.2, seed=2)
    f = np.random.default_rng(4).uniform(-1, 1, p.n_dof)
    ctx = FemContext(p, semantics="consistent")
    assert ctx.diagonal().min() > 2e5  # (r.z < 5e-46: below half the smallest FP32 number, 1.4e-45)
    u, info = ctx.pcg(1e-20 * f, precision="fp32_refine", tol=tol, stop_rule=rule, outer_tol=1e-9)
    assert (info["status"], info["iterations"], info["outer_iterations"]) == (0, 0, 2)
    assert not u.any() and info["rel_residual"] == 1.0
    u, info = ctx.pcg(f, precision="fp32_refine", tol=tol, stop_rule=rule, outer_tol=1e-11)
    x, _ = O.Oracle(p, consistent=True).assemble().pcg(f, tol=1e-14, rule=1)
    assert info["rel_residual"] <= 1e-11 and rel(u, x) <= 1e-7


@pytest.mark.parametrize("load", ["end", "random"])
def test_refinement_of_a_slender_beam(load):
    """A beam 300 cells long: ten thousand FP32 iterations per refinement step and
    more, in which the residual first rises far above its start; whole runs need
    0.11 to 0.13 M in all, runs cut after 512 0.5 to 1.4 M, and capped at 20000 per
    step they end as converged at residuals of 0.3 to 2. A solve that says it has
    converged to 1e-6 has: f - K u from the elements, in displacement differences."""
    from cudafemproject_gb300.solver import FemContext
    p = meshgen.box_3d(1, 1, 300, lz=300.0, jitter=0.2, seed=0)
    f = np.random.default_rng(5).standard_normal((p.n_nodes, 3))
    if load == "end":
        f[p.nodes[:, 2] < 0.95 * p.nodes[:, 2].max()] = 0
    f[p.cons[:, 0]] = 0
    f = f.ravel()
    ctx = FemContext(p, semantics="consistent")
    _, info = ctx.pcg(f, precision="fp32_refine", tol=1e-3, stop_rule="residual", outer_tol=1e-6, max_iter=20000,
                      allow_not_converged=True)
    assert info["status"] != 0 or info["rel_residual"] <= 1e-6
    u, info = ctx.pcg(f, precision="fp32_refine", tol=1e-3, stop_rule="residual", outer_tol=1e-6)
    assert info["rel_residual"] <= 1e-6 and info["iterations"] <= 300000
    X, U = p.nodes[p.elems], u.reshape(-1, 3)[p.elems]
    J = X[:, 1:] - X[:, :1]
    g = np.linalg.inv(J).transpose(0, 2, 1)  # gradients of N_1 .. N_3 (U is zero at the clamped nodes)
    H = np.einsum("eai,eaj->eij", U[:, 1:] - U[:, :1], g)
    lam, mu = p.E * p.nu / ((1 + p.nu) * (1 - 2 * p.nu)), p.E / (2 * (1 + p.nu))
    S = lam * np.trace(H, axis1=1, axis2=2)[:, None, None] * np.eye(3) + mu * (H + H.transpose(0, 2, 1))
    F = np.einsum("eij,eaj->eai", S, g) * (np.abs(np.linalg.det(J)) / 6)[:, None, None]
    r = f.copy().reshape(-1, 3)
    np.subtract.at(r, p.elems[:, 1:], F)
    np.add.at(r, p.elems[:, 0], F.sum(1))
    r[p.cons[:, 0]] = 0
    assert np.linalg.norm(r) <= 1.5e-6 * np.linalg.norm(f)


def test_fp64_steps_of_contexts_in_several_threads():
    """Explicit FP64 steps with re-sorted masses (96 KB of dynamic shared memory) and
    with constant ones (none) are the same kernel. Contexts of both kinds that step
    in threads of their own get what each gets alone."""
    import ctypes as C
    import threading
    from cudafemproject_gb300 import capi
    from cudafemproject_gb300.solver import FemContext
    p = meshgen.box_3d(2, 2, 3, jitter=0.2, seed=2, rho=2000.0, traction=None, point_load=("top_centre", (0.4, -0.3, -1.0)))
    ctxs = [FemContext(p, semantics=k) for k in ("compat", "consistent", "consistent")]
    alone = [c.dyn(0.5, 0.0, 1e-5, 3e-5 * 1.0000001, precision="fp64")[0].ravel() for c in ctxs]
    wrong = []

    def steps(c, want):
        u, inf = np.zeros(p.n_dof), capi.DynInfo()
        prm = capi.DynParams(0.5, 0.0, 1e-5, 3e-5 * 1.0000001, capi.FP64, 0.0, 0, 0, 0, 0, None, None)
        for _ in range(6000):
            st = capi.lib().cfem_dyn(c._h, C.byref(prm), None, u.ctypes.data, C.byref(inf))
            if st != capi.OK:
                wrong.append(capi.lib().cfem_last_error_string())
            elif not np.array_equal(u, want):
                wrong.append("another result")

    threads = [threading.Thread(target=steps, args=a) for a in zip(ctxs, alone)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, (len(wrong), wrong[0])


def test_geometry_contexts_of_several_patch_sizes():
    """The shared memory that a geometry-form context needs does not depend on the
    contexts created after it."""
    from cudafemproject_gb300.solver import FemContext
    p = meshgen.box_3d(8, 8, 16, jitter=0.2, seed=2)
    x = np.random.default_rng(1).standard_normal(p.n_dof).astype(np.float32)
    large = FemContext(p, semantics="consistent", matvec_form="geometry", patch_elems=768)
    y = large.matvec(x, precision="fp32")
    small = FemContext(p, semantics="consistent", matvec_form="geometry", patch_elems=64)
    # (FP32 sums of up to a hundred terms in another order)
    assert rel(small.matvec(x, precision="fp32"), y) <= 1e-5
    assert rel(large.matvec(x, precision="fp32"), y) <= 1e-5


def _column():
    return meshgen.box_3d(4, 3, 17, lz=4.0, jitter=0.2, seed=5, rho=2000.0, traction=None,
                          point_load=("top_centre", (0.4, -0.3, -1.0)))


def _implicit(ctx, p, precision, n, cap, rec):
    """Status, displacements, trace and PCG iterations of n implicit steps with at most cap iterations each."""
    import ctypes as C
    from cudafemproject_gb300 import capi
    u, trace = np.full(p.n_dof, np.nan), np.full((n, len(rec), 3), np.nan)
    prm = capi.DynParams(0.5, 0.5, 1e-3, n * 1e-3 * 1.0000001, {"fp64": capi.FP64, "fp32": capi.FP32}[precision], 1e-6,
                         capi.STOP_RESIDUAL, cap, 1, len(rec), rec.ctypes.data, trace.ctypes.data)
    inf = capi.DynInfo()
    st = capi.lib().cfem_dyn(ctx._h, C.byref(prm), None, u.ctypes.data, C.byref(inf))
    return st, u.reshape(-1, 3), trace, inf.pcg_iterations


@pytest.mark.parametrize("host_loop", [False, True])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_implicit_trace_and_failing_step(monkeypatch, precision, host_loop):
    """Row n of an implicit run's receiver trace is the displacement that a run of n
    steps ends with (FP32 sums are atomic: 1e-5), on a context that has run before.
    Where step s does not converge, the rows before it are those, u is the state
    before it and the rows from s on are zero: not what the kept buffers held."""
    from cudafemproject_gb300 import capi
    from cudafemproject_gb300.solver import FemContext
    if host_loop:
        monkeypatch.setenv("CFEM_HOST_LOOP", "1")
    else:
        monkeypatch.delenv("CFEM_HOST_LOOP", raising=False)
    p = _column()
    ctx = FemContext(p, semantics="consistent")
    rec = np.array([int(p.load_node[0]), p.n_nodes - 1, p.n_nodes // 2], np.int32)
    ends, its = [np.zeros((p.n_nodes, 3))], [0]
    for n in range(1, 7):
        st, u, trace, k = _implicit(ctx, p, precision, n, 1000, rec)
        assert st == capi.OK
        ends.append(u)
        its.append(k)
        for i in range(n):
            assert rel(trace[i], ends[i + 1][rec]) <= 1e-5
        assert np.array_equal(trace[-1], u[rec])
    need = np.diff(its)
    for cap in sorted({int(need[0]), int(need.max()) - 1, 1}):
        bad = next((i for i, k in enumerate(need) if k > cap), None)
        if bad is None:
            continue
        st, u, trace, _ = _implicit(ctx, p, precision, 6, cap, rec)
        assert st == capi.ERR_NOT_CONVERGED
        assert rel(u, ends[bad]) <= 1e-5 if bad else not u.any()
        for i in range(bad):
            assert rel(trace[i], ends[i + 1][rec]) <= 1e-5
        assert not trace[bad:].any()


def test_implicit_step_queued_behind_a_failing_one_takes_no_iteration():
    """FP32 implicit steps are queued one ahead. Where a step ends at its iteration
    cap (large steps: hundreds of iterations), the one behind it takes none: a run
    of six steps that fails in its first takes the time of that step, not of two."""
    import ctypes as C
    import time
    from cudafemproject_gb300 import capi
    from cudafemproject_gb300.solver import FemContext
    p = meshgen.box_3d(3, 3, 60, lz=20.0, jitter=0.2, seed=5, rho=2000.0, traction=None, point_load=("top_centre", (0.4, -0.3, -1.0)))
    ctx = FemContext(p, semantics="consistent")
    cap = 250

    def failing(n):
        u, inf = np.zeros(p.n_dof), capi.DynInfo()
        prm = capi.DynParams(0.5, 0.5, 10.0, n * 10.0 * 1.0000001, capi.FP32, 1e-6, capi.STOP_RESIDUAL, cap, 1, 0, None, None)
        t = time.perf_counter()
        st = capi.lib().cfem_dyn(ctx._h, C.byref(prm), None, u.ctypes.data, C.byref(inf))
        t = time.perf_counter() - t
        assert st == capi.ERR_NOT_CONVERGED and inf.pcg_iterations == cap and not u.any()
        return t

    one, six = (sorted(failing(n) for _ in range(15))[7] for n in (1, 6))
    # (with the whole step behind it 2.0; with its other kernels and one loop body 1.1)
    assert six <= 1.4 * one


def test_multi_rhs_iteration_cap_holds_per_step():
    """Load cases that need few and many iterations, a loose inner tolerance: the
    steps of the slow ones go on over several rounds, and max_iter holds for a
    step, not for each of its rounds."""
    from cudafemproject_gb300.solver import FemContext
    p = meshgen.box_3d(3, 3, 40, jitter=0.2, seed=2)
    rng = np.random.default_rng(3)
    F = rng.standard_normal((8, p.n_dof))
    top = p.nodes[:, 2] > p.nodes[:, 2].max() - 1e-6
    F[:2] = 0
    F[0].reshape(-1, 3)[top] = (1.0, 0.0, 0.0)  # bending: the slow modes only
    F[1].reshape(-1, 3)[top] = (0.0, 1.0, 0.0)
    ctx = FemContext(p, semantics="consistent")
    for cap in (20, 35, 50, 75, 100, 150, 200, 300):
        _, infos = ctx.pcg_multi(F, precision="fp32_refine", tol=0.3, stop_rule="residual", outer_tol=1e-9, max_iter=cap,
                                 max_outer=12, allow_not_converged=True)
        for i in infos:
            assert i["iterations"] <= cap * max(1, i["outer_iterations"]), (cap, i)


def test_dyn_adjoint_without_room_for_all_states():
    """481 MB of states within the 1 GB limit, on a device with 250 MB left: the
    reverse sweep goes by segments, with the loss and gradient of the whole sweep
    (the steps are taken again with the same sums)."""
    import torch
    from cudafemproject_gb300.solver import FemContext
    p = meshgen.box_3d(16, 16, 64, jitter=0.2, seed=5, rho=2000.0, traction=None, point_load=("top_centre", (0.4, -0.3, -1.0)))
    ctx = FemContext(p, semantics="consistent")
    rec = np.array([int(p.load_node[0]), p.n_nodes - 1], np.int32)
    args = (0.5, 1e-5, 400e-5 * 1.0000001, rec, 1e-9 * np.random.default_rng(1).standard_normal((400, 2, 3)))
    torch.cuda.empty_cache()
    hog = []
    try:
        for keep in (8 << 30, 1 << 30, 250 << 20):  # (in a few pieces: the free memory need not be one)
            free = torch.cuda.mem_get_info()[0]
            if free > keep:
                hog.append(torch.empty((free - keep) // (2 << 20) * (2 << 20), dtype=torch.uint8, device="cuda"))
        left = torch.cuda.mem_get_info()[0]
        assert left < 2 * 401 * 4 * p.n_nodes * 8
        by_segments = ctx.dyn_adjoint(*args)
    finally:
        del hog
        torch.cuda.empty_cache()
    whole = FemContext(p, semantics="consistent").dyn_adjoint(*args)
    assert by_segments[0] == pytest.approx(whole[0], rel=1e-12)
    assert rel(by_segments[1], whole[1]) <= 1e-12


def _hub(n_rim):
    """A double cone of tetrahedra around one axis edge, which all of them share."""
    from cudafemproject_gb300.meshio import Problem
    t = 2 * np.pi * np.arange(n_rim) / n_rim
    nodes = np.concatenate([[[0, 0, -1], [0, 0, 1]], np.stack([np.cos(t), np.sin(t), 0.1 * np.cos(3 * t)], axis=1)])
    i, z = np.arange(n_rim), np.zeros((0, 3))
    elems = np.stack([np.zeros_like(i), np.ones_like(i), 2 + i, 2 + (i + 1) % n_rim], axis=1)
    return Problem(dim=3, nodes=nodes.astype(np.float32).astype(np.float64), elems=elems.astype(np.int32),
                   cons=np.array([[2, 7], [5, 1], [9, 2], [1, 4]], np.int32), load_node=np.zeros(0, np.int32), load_vec=z,
                   face_nodes=np.zeros((0, 4), np.int32), face_elem=np.zeros(0, np.int32), face_normal=z,
                   face_pressure=np.zeros(0), E=2e7, nu=0.25, rho=2000.0, elem_E=None)


@pytest.mark.parametrize("n_rim", [31, 64, 65, 96, 97, 98, 128, 129, 1000, 4001])
def test_nodes_of_many_elements(n_rim):
    """Two nodes with n_rim + 1 neighbours and an edge that n_rim elements share (and
    the limits from which a warp works on such a row and edge): products, diagonal
    and a solve against the oracle, after new moduli, too. (A row of n products of
    random signs rounds by sqrt(n) units and their sum may cancel: 1e-12. Solves to
    a residual of 1e-13 differ by the condition number times that, (n_rim / 2 pi)^2
    and a factor of hundreds for these needles: up to 129 of them.)"""
    from cudafemproject_gb300.solver import FemContext
    p = _hub(n_rim)
    ctx = FemContext(p, semantics="consistent")
    rng = np.random.default_rng(n_rim)
    for young in (None, 2e7 * np.exp(0.3 * rng.standard_normal(p.n_elems))):
        if young is not None:
            ctx.set_young(young)
            p.elem_E = young
        o = O.Oracle(p, consistent=True)
        x = rng.standard_normal(p.n_dof)
        assert rel(ctx.matvec(x, "fp64"), o.matvec(x)) <= 1e-12
    if n_rim <= 129:
        f = rng.standard_normal(p.n_dof)
        xo, _ = o.pcg(f, tol=1e-13, rule=1)
        assert rel(ctx.pcg(f, "fp64", tol=1e-13, stop_rule="residual")[0], xo) <= 1e-8
        for u in ctx.pcg_multi(np.stack([f, 2 * f]), "fp32_refine", tol=0.3, stop_rule="residual", outer_tol=1e-11)[0]:
            assert min(rel(u, xo), rel(u, 2 * xo)) <= 1e-7


def test_moduli_of_nodes_of_many_elements_take_linear_time():
    """set_young on a node of m elements: sixteen times the elements in less than
    forty times the time (a scan of them for each neighbour: 256 times)."""
    import time
    from cudafemproject_gb300.solver import FemContext

    def seconds(n):
        ctx, y, ts = FemContext(_hub(n)), np.full(n, 2e7), []
        for _ in range(9):
            t = time.perf_counter()
            ctx.set_young(y)
            ts.append(time.perf_counter() - t)
        return sorted(ts)[4]

    assert seconds(8000) <= 40 * seconds(500)


@pytest.mark.parametrize("semantics", ["consistent", "compat"])
@pytest.mark.parametrize("n_rim", [63, 64, 65, 300])
def test_steps_with_nodes_of_many_elements(n_rim, semantics):
    """Explicit and implicit FP64 steps and the steps' adjoint on rows of their own
    slices (n_rim + 1 neighbours each, the limit is 64), against the oracle and a
    central difference of the loss."""
    from cudafemproject_gb300.solver import FemContext
    p = _hub(n_rim)
    p.load_node, p.load_vec = np.array([0, 40], np.int32), np.array([[0.1, 0.2, -1.0], [1.0, 0.0, 0.5]])
    dt, rec = 1e-6, np.array([0, 1, 50], np.int32)
    ctx, o = FemContext(p, semantics=semantics), O.Oracle(p, consistent=semantics == "consistent")
    for steps in (1, 5):
        ug, st, _ = o.dyn(0.5, 0.0, dt, steps * dt * 1.0000001)
        u, _, trace = ctx.dyn(0.5, 0.0, dt, steps * dt * 1.0000001, precision="fp64", receivers=rec)
        # (a few steps with other summation orders, rows of n_rim products)
        assert rel(u, ug) <= 1e-10 and np.array_equal(trace[-1], u[rec])
    if semantics == "consistent":
        obs = np.zeros((4, 3, 3))
        young = np.full(p.n_elems, p.E)
        loss, g, _ = ctx.dyn_adjoint(0.5, dt, 4 * dt * 1.0000001, rec, obs)
        d = young * np.random.default_rng(1).standard_normal(p.n_elems) * 1e-4
        ends = []
        for s in (1, -1):
            ctx.set_young(young + s * d)
            ends.append(ctx.dyn_adjoint(0.5, dt, 4 * dt * 1.0000001, rec, obs)[0])
        # (the loss is smooth in the moduli: the difference's error is of order 1e-8)
        assert (ends[0] - ends[1]) / 2 == pytest.approx(float(g @ d), rel=1e-5, abs=1e-9 * abs(loss))


@pytest.mark.parametrize("mesh", ["box", "large", "plate", "hub"])
def test_missing_cta_is_reported_and_context_recovers(mesh):
    """The failure path of the cooperative FP64 kernels' exchanges, without a fault:
    each is launched without its CTA 0, with waits bounded at ~1 ms. The others
    give up and return, the host reports it, and the context then works: rows in
    registers, in memory (more slices than warps), 2D, rows of a warp."""
    from cudafemproject_gb300 import capi
    from cudafemproject_gb300.solver import FemContext
    p = {"box": lambda: meshgen.box_3d(6, 6, 18, jitter=0.2, seed=2), "large": lambda: meshgen.box_3d(24, 24, 72, jitter=0.2, seed=2),
         "plate": lambda: meshgen.square_2d(30), "hub": lambda: _hub(120)}[mesh]()
    ctx = FemContext(p, semantics="consistent")
    L = capi.lib()
    for _ in range(2):
        assert L.cfem_selftest_grid_timeout(ctx._h) == capi.OK, L.cfem_last_error_string()
    x = np.random.default_rng(1).standard_normal(p.n_dof)
    f = ctx.matvec(x, "fp64")
    u, info = ctx.pcg(f, "fp64", tol=1e-10, stop_rule="residual")
    # (the residual's floor, and the condition number in front of the difference)
    assert info["status"] == 0 and info["rel_residual"] <= 1e-9
    ud, info = ctx.dyn(0.5, 0.0, 1e-9, 3.0000003e-9, precision="fp64")
    assert info["steps"] == 3 and np.isfinite(ud).all()
    assert L.cfem_selftest_grid_timeout(FemContext(meshgen.square_2d(4), semantics="consistent")._h) == capi.ERR_UNSUPPORTED


@pytest.mark.parametrize("form", ["auto", "geometry", "gradient"])
@pytest.mark.parametrize("semantics", ["consistent", "compat"])
@pytest.mark.parametrize("beta2", [0.0, 0.5])
def test_fp32_traces_row_by_row(beta2, semantics, form):
    """FP32 steps on a mesh of one patch, where no sum depends on the order of atomic
    additions: row n of the receiver trace is the displacement that n steps end
    with, bit by bit, on a fresh context as on one that has run before with another
    context's run in between."""
    from cudafemproject_gb300.meshio import WaveletParams
    from cudafemproject_gb300.solver import FemContext
    p = meshgen.box_3d(3, 3, 8, jitter=0.2, seed=5, rho=2000.0, traction=None, point_load=("top_centre", (0.4, -0.3, -1.0)))
    dt = 2e-5 if beta2 == 0 else 1e-3
    rec = np.array([int(p.load_node[0]), p.n_nodes - 1, p.n_nodes // 2], np.int32)
    w = WaveletParams("ricker", 40.0, 0.0, 1.0)

    def run(ctx, n):
        return ctx.dyn(0.5, beta2, dt, n * dt * 1.0000001, precision="fp32", wavelet=w, pcg_tol=1e-6, receivers=rec)

    ctx, other = (FemContext(p, semantics=semantics, matvec_form=form) for _ in range(2))
    assert ctx.counts()["n_patches"] == 1
    N = 15
    u, _, trace = run(ctx, N)
    assert np.array_equal(trace[-1], u[rec]) and trace.any()
    for n in range(1, N + 1):
        un, _, tn = run(ctx, n)
        assert np.array_equal(un[rec], trace[n - 1]) and np.array_equal(tn, trace[:n]), n
        run(other, 4)
    assert np.array_equal(run(ctx, N)[0], u)


@pytest.mark.parametrize("side", ["largest", "smallest"])
@pytest.mark.parametrize("limit", [4, 16])
def test_fp64_pcg_shapes_on_either_side_of_their_limits(limit, side):
    """The one-kernel PCG has at most four slices of 16 rows per CTA (128 threads), at
    most sixteen (512), or more: plates with the most nodes on one side of a limit
    on this GPU and the fewest on the other, and some tens of CTAs of the first
    kind. Iterates 1 and 2 (two recurrences that differ in the order of their sums:
    1e-12) and a converged solve (1e-10, the bar of every FP64 solve)."""
    import torch
    from cudafemproject_gb300.solver import FemContext
    slices = limit * torch.cuda.get_device_properties(0).multi_processor_count
    n = max(n for n in range(2, 400) if -(-(n + 1) ** 2 // 16) <= slices) + (side == "smallest")
    for m in {n, 40 if (limit, side) == (4, "largest") else n}:
        p = meshgen.square_2d(m)
        f = np.zeros((p.n_nodes, 2))
        f[p.nodes[:, 0] > 1 - 1e-9] = (0.7, -0.2)
        f = f.ravel()
        ctx, o = FemContext(p, semantics="consistent"), O.Oracle(p, consistent=True)
        for iters in (1, 2):
            x, it = o.pcg(f, tol=1e-30, rule=1, maxit=iters, allow_maxit=True)
            u, info = ctx.pcg(f, "fp64", tol=1e-30, stop_rule="residual", max_iter=iters, allow_not_converged=True)
            assert info["iterations"] == it == iters and rel(u, x) <= 1e-12
        u, _ = ctx.pcg(f, "fp64", tol=1e-13, stop_rule="residual")
        assert rel(u, o.pcg(f, tol=1e-13, rule=1)[0]) <= 1e-10


def _fan(n):
    """A fan of n triangles around one node."""
    from cudafemproject_gb300.meshio import Problem
    t = 2 * np.pi * np.arange(n) / n
    nodes = np.concatenate([[[0.0, 0.0]], np.stack([np.cos(t), np.sin(t)], axis=1)])
    i, z = np.arange(n), np.zeros((0, 2))
    return Problem(dim=2, nodes=nodes.astype(np.float32).astype(np.float64),
                   elems=np.stack([np.zeros_like(i), 1 + i, 1 + (i + 1) % n], axis=1).astype(np.int32),
                   cons=np.array([[1, 3], [4, 1], [7, 2]], np.int32), load_node=np.array([0, n // 2], np.int32),
                   load_vec=np.array([[0.3, -1.0], [0.5, 0.2]]), face_nodes=np.zeros((0, 3), np.int32),
                   face_elem=np.zeros(0, np.int32), face_normal=z, face_pressure=np.zeros(0), E=2e7, nu=0.25, rho=2000.0,
                   elem_E=None)


@pytest.mark.parametrize("body", ["fan64", "fan65", "fan300", "hub64", "hub120"])
def test_rows_of_a_warp_in_every_fp64_call(body):
    """Nodes of 64, 65 and more neighbours in 2D and 3D: products, a solve, explicit
    steps and implicit ones (stiffness and mass in the same blocks) against the
    oracle. (Products and a few explicit steps: rows of up to 300 terms, 1e-12 and
    1e-10; a solve to 1e-13 and implicit steps whose PCG stops at 1e-12: the
    condition number of the needles in front, up to 1e4, and two solvers: 1e-8.)"""
    from cudafemproject_gb300.solver import FemContext
    n = int(body[3:])
    p = _fan(n) if body.startswith("fan") else _hub(n)
    if body.startswith("hub"):
        p.load_node, p.load_vec = np.array([0, 40], np.int32), np.array([[0.1, 0.2, -1.0], [1.0, 0.0, 0.5]])
    ctx, o = FemContext(p, semantics="consistent"), O.Oracle(p, consistent=True)
    x = np.random.default_rng(n).standard_normal(p.n_dof)
    assert rel(ctx.matvec(x, "fp64"), o.matvec(x)) <= 1e-12
    f = o.matvec(x)
    assert rel(ctx.pcg(f, "fp64", tol=1e-13, stop_rule="residual")[0], o.pcg(f, tol=1e-13, rule=1)[0]) <= 1e-8
    for beta2, dt in ((0.0, 1e-7), (0.5, 1e-5)):
        ug, st, _ = o.dyn(0.5, beta2, dt, 3 * dt * 1.0000001, **({} if beta2 == 0 else dict(pcg_tol=1e-12)))
        u, info = ctx.dyn(0.5, beta2, dt, 3 * dt * 1.0000001, precision="fp64", pcg_tol=1e-12)
        assert info["steps"] == st == 3
        assert rel(u, ug) <= (1e-10 if beta2 == 0 else 1e-8)
