"""FP32 solves with FP64 refinement: steps of several FP32 runs ("legs"), against
the FP64 oracle."""
import numpy as np
import pytest

import oracle as O
from conftest import rel
from cudafemproject_gb300 import meshgen

pytestmark = pytest.mark.gpu


MESHES = {
    "box": lambda: meshgen.box_3d(6, 5, 21, jitter=0.2, seed=3),
    "beam": lambda: meshgen.box_3d(2, 2, 90, jitter=0.2, seed=5),  # most iterations per leg
    "plate": lambda: meshgen.square_2d(17),
    "tets": lambda: meshgen.random_tets(900),
}


@pytest.mark.parametrize("host_loop", [False, True])
@pytest.mark.parametrize("rule", ["residual", "reference"])
@pytest.mark.parametrize("mesh", sorted(MESHES))
def test_refinement_legs(monkeypatch, mesh, rule, host_loop):
    """Inner tolerances down from a leg's: the outer tolerance is met and the solution
    is the oracle's. Legs do not count as steps: one per factor of the inner
    tolerance, and two for what a step may lose to rounding."""
    from cudafemproject_gb300.solver import FemContext
    if host_loop:
        monkeypatch.setenv("CFEM_HOST_LOOP", "1")
    else:
        monkeypatch.delenv("CFEM_HOST_LOOP", raising=False)
    p = MESHES[mesh]()
    f = np.random.default_rng(1).standard_normal(p.n_dof)
    x, _ = O.Oracle(p, consistent=True).assemble().pcg(f, tol=1e-14, rule=1)
    ctx = FemContext(p, semantics="consistent")
    for tol in (0.1, 0.03, 1e-3, 1e-6):
        u, info = ctx.pcg(f, precision="fp32_refine", tol=tol, stop_rule=rule, outer_tol=1e-11)
        assert info["status"] == 0 and info["rel_residual"] <= 1e-11
        # (the condition number times the residual: about 1e4, of the beam (45 long) 45^4)
        assert rel(u, x) <= (1e-4 if mesh == "beam" else 1e-7)
        if rule == "residual":  # (a sixteenth of the outer tolerance: 12.2 digits)
            assert info["outer_iterations"] <= np.ceil(12.2 / -np.log10(tol)) + 2


def test_refinement_legs_limits():
    """One refinement step ends at its tolerance, an iteration cap holds per step (a
    cap of 7 and of 600, more than one leg), and an outer tolerance below the FP64
    floor ends as converged at the floor."""
    from cudafemproject_gb300.solver import FemContext
    p = MESHES["beam"]()
    f = np.random.default_rng(2).standard_normal(p.n_dof)
    ctx = FemContext(p, semantics="consistent")
    kw = dict(precision="fp32_refine", stop_rule="residual", allow_not_converged=True)
    u, one = ctx.pcg(f, tol=1e-3, outer_tol=1e-11, max_outer=1, **kw)
    assert one["status"] != 0 and one["outer_iterations"] == 1
    # (the recurrence met 1e-3; a leg may have drifted off by up to 1.1 before it was replaced)
    assert one["rel_residual"] <= 2e-3
    for cap in (7, 600):
        u, info = ctx.pcg(f, tol=1e-6, outer_tol=1e-11, max_iter=cap, max_outer=1, **kw)
        assert info["outer_iterations"] == 1 and info["iterations"] <= cap
    assert info["iterations"] == cap or info["rel_residual"] <= 1e-5
    u, info = ctx.pcg(f, tol=1e-3, outer_tol=1e-20, max_outer=60, **kw)
    assert info["status"] == 0 and info["rel_residual"] <= 1e-11 and info["outer_iterations"] < 60
