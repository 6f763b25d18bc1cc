"""The single-launch solvers (``femk_persist.cu``) against the chunked ones on the same system.

``femk_pcg`` runs systems whose operator stays on the chip as one launch: one block, one cluster, or a
cooperative grid, by size. A plan whose options name a kernel of the chunked solver (``ring64`` = 14, its
default) keeps that solver, which the other tests hold to the oracle. Both run the same operations but for the
order of the dot products, so their iterates agree to rounding: at relative residuals of 1e-10 and these
condition numbers (below 1e5) to far less than 1e-9 unless the stop test falls on another iteration, and then by
one step, itself below the residual bound times the condition number's root: 1e-7 covers both."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import mesh as om  # noqa: E402


def _mesh(dim, n, order, shuffled, seed=5):
    from jno_b200.domain import box_points_tets, jitter_interior, jitter_interior_2d, rect_points_tris

    if dim == 3:
        pts, cells = box_points_tets(*n)
        pts = jitter_interior(pts, *n, seed=seed)
    else:
        pts, cells = rect_points_tris(*n)
        pts = jitter_interior_2d(pts, *n, seed=seed)[:, :2]
    if shuffled:
        rng = np.random.default_rng(seed)
        perm = rng.permutation(len(pts))
        moved = np.empty_like(pts)
        moved[perm] = pts
        pts, cells = moved, perm[cells][rng.permutation(len(cells))]
    return pts, cells


def _plans(dim, n, order, shuffled):
    from jno_b200.plan import FemPlan

    pts, cells = _mesh(dim, n, order, shuffled)
    one, chunked = FemPlan(pts, cells, order), FemPlan(pts, cells, order, options={"ring64": 14})
    logk = torch.as_tensor(om.logk_field(len(cells), 1015), device="cuda")
    vals, b = one.assemble(logk)
    return one, chunked, vals, b, one.jacobi(vals)


# (dim, cells per axis, order, shuffled): one block (a single row of slices, its largest size), the smallest
# cluster, 16 blocks of 32 slices (n = 16,384), one row past that (the grid), a grid of all SMs, 2-D rows of at
# most 9 entries, P2's unequal rows with int32 columns, and vertices in no order
SYSTEMS = [
    (3, (2, 2, 2), 1, False),
    (3, (9, 9, 10), 1, False),
    (3, (10, 10, 11), 1, False),
    (2, (127, 127), 1, False),
    (2, (128, 126), 1, False),
    (2, (128, 127), 1, False),
    (3, (33, 35, 31), 1, False),
    (3, (44, 43, 47), 1, False),
    (3, (5, 6, 7), 2, False),
    (3, (17, 13, 15), 2, False),
    (2, (75, 61), 2, False),
    (3, (21, 23, 22), 1, True),
    (2, (40, 33), 2, True),
]


@pytest.mark.parametrize("dim,n,order,shuffled", SYSTEMS)
@pytest.mark.parametrize("precond", [True, False])
def test_pcg_matches_the_chunked_solver(dim, n, order, shuffled, precond):
    one, chunked, vals, b, inv = _plans(dim, n, order, shuffled)
    inv = inv if precond else None
    g = torch.Generator(device="cuda").manual_seed(1)
    start = torch.randn(one.n, dtype=torch.float64, device="cuda", generator=g) * b.abs().max()
    for x0 in (torch.zeros_like(b), start):
        x, it, rel, st = one.pcg(vals, b, x0.clone(), inv, tol=1e-10)
        y, ity, rely, sty = chunked.pcg(vals, b, x0.clone(), inv, tol=1e-10)
        assert st == 0 and sty == 0
        if precond:  # without one the chunked solver's own kernels differ by up to two iterations in 2-D
            assert abs(it - ity) <= 1, (it, ity)
        assert abs(rel - (torch.linalg.norm(b - one.spmv(vals, x)) / torch.linalg.norm(b)).item()) <= 1e-12
        assert (torch.linalg.norm(x - y) / torch.linalg.norm(y)).item() <= 1e-7
        again, it2, rel2, _ = one.pcg(vals, b, x0.clone(), inv, tol=1e-10)
        assert it2 == it and rel2 == rel and torch.equal(again, x)


@pytest.mark.parametrize("dim,n,order", [(3, (3, 3, 3), 1), (3, (14, 14, 14), 1), (3, (33, 35, 31), 1)])
def test_pcg_status_paths_match_the_chunked_solver(dim, n, order):
    """The iteration cap, no iteration at all, a zero load, a non-finite load and an indefinite operator give the
    status, the iteration count and the iterate of the chunked solver."""
    from jno_b200 import _lib

    one, chunked, vals, b, inv = _plans(dim, n, order, False)
    for maxiter in (0, 1, 7):
        got = [p.pcg(vals, b, None, inv, 1e-12, maxiter=maxiter) for p in (one, chunked)]
        assert got[0][3] == got[1][3] and got[0][1] == got[1][1] == maxiter
        assert torch.allclose(got[0][0], got[1][0], rtol=0, atol=1e-12 * max(1e-300, got[1][0].abs().max().item()))
    x, it, rel, st = one.pcg(vals, torch.zeros_like(b), None, inv)
    assert (it, st, rel) == (0, 0, 0.0) and torch.all(x == 0)
    bad = b.clone()
    bad[one.n // 2] = float("nan")
    for load, v in ((bad, vals), (b, -vals)):
        codes = []
        for p in (one, chunked):
            with pytest.raises(_lib.FemkError) as e:
                p.pcg(v, load, None, inv)
            codes.append(str(e.value))
        assert codes[0] == codes[1]
    x, it, rel, st = one.pcg(vals, b, None, inv)  # and the plan goes on
    assert st == 0 and rel <= 2e-8


def test_a_grid_wait_that_runs_out_is_a_status():
    """Block 0 never arrives at the grid's first sum: every block gives up after the limit, the call reports it,
    and the next plan solves on the same device."""
    from jno_b200 import _lib
    from jno_b200.plan import FemPlan

    pts, cells = _mesh(3, (33, 35, 31), 1, False)
    plan = FemPlan(pts, cells, 1, options={"test_skip_arrival": 0, "barrier_limit_ms": 5.0})
    vals, b = plan.assemble(torch.zeros(len(cells), dtype=torch.float64, device="cuda"))
    inv = plan.jacobi(vals)
    for _ in range(2):
        with pytest.raises(_lib.FemkError, match="wait"):
            plan.pcg(vals, b, None, inv)
    x, it, rel, st = FemPlan(pts, cells, 1).pcg(vals, b, None, inv)
    assert st == 0 and rel <= 2e-8


@pytest.mark.parametrize("dim,n,order,shuffled", SYSTEMS)
@pytest.mark.parametrize("precond", [True, False])
def test_bicgstab_matches_the_chunked_solver(dim, n, order, shuffled, precond):
    """BiCGStab's count moves with the order of its sums, so the solutions are held to each other: both meet a
    relative residual of 1e-11, which bounds their distance by twice that times the condition number (below 1e5
    here, without a preconditioner too): 2e-6."""
    one, chunked, vals, b, inv = _plans(dim, n, order, shuffled)
    inv = inv if precond else None
    g = torch.Generator(device="cuda").manual_seed(2)
    start = torch.randn(one.n, dtype=torch.float64, device="cuda", generator=g) * b.abs().max()
    for x0 in (torch.zeros_like(b), start):
        x, it, rel, st = one.bicgstab(vals, b, x0.clone(), inv, tol=1e-11)
        y, _, _, sty = chunked.bicgstab(vals, b, x0.clone(), inv, tol=1e-11)
        assert st == sty == 0
        assert abs(rel - (torch.linalg.norm(b - one.spmv(vals, x)) / torch.linalg.norm(b)).item()) <= 1e-12
        assert (torch.linalg.norm(x - y) / torch.linalg.norm(y)).item() <= 2e-6
        again, it2, rel2, _ = one.bicgstab(vals, b, x0.clone(), inv, tol=1e-11)
        assert it2 == it and rel2 == rel and torch.equal(again, x)


@pytest.mark.parametrize("dim,n,order", [(3, (3, 3, 3), 1), (3, (14, 14, 14), 1), (3, (33, 35, 31), 1)])
def test_bicgstab_status_paths_match_the_chunked_solver(dim, n, order):
    from jno_b200 import _lib

    one, chunked, vals, b, inv = _plans(dim, n, order, False)
    for maxiter in (0, 1, 3):
        got = [p.bicgstab(vals, b, None, inv, 1e-12, maxiter=maxiter) for p in (one, chunked)]
        assert got[0][3] == got[1][3] and got[0][1] == got[1][1] == maxiter
        assert torch.allclose(got[0][0], got[1][0], rtol=0, atol=1e-11 * max(1e-300, got[1][0].abs().max().item()))
    bad = b.clone()
    bad[one.n // 2] = float("nan")
    for p in (one, chunked):
        with pytest.raises(_lib.FemkError, match="non-finite"):
            p.bicgstab(vals, bad, None, inv)


@pytest.mark.parametrize("dim,n,order", [(2, (19, 23), 1), (3, (14, 13, 15), 1), (3, (33, 35, 31), 1), (3, (9, 8, 7), 2)])
def test_theta_march_matches_the_chunked_solver(dim, n, order):
    """Every step to 1e-12 of its right-hand side; the step systems' condition numbers are below 1e3 at this dt:
    1e-8 of the state's size covers the steps together."""
    from jno_b200.plan import FemPlan

    pts, cells = _mesh(dim, n, order, False)
    logk = torch.as_tensor(om.logk_field(len(cells), 1016), device="cuda")
    states = []
    for options in (None, {"ring64": 14}):
        plan = FemPlan(pts, cells, order, options=options)
        S, R, q = plan.assemble_theta(logk, theta=0.5, dt=1e-3)
        u = plan.lumped_mass() / plan.lumped_mass().abs().max()
        u, _, worst = plan.theta_march(S, R, q, u, 5, tol=1e-12)
        assert worst <= 1e-11
        states.append(u)
    assert (states[0] - states[1]).abs().max() <= 1e-8 * states[1].abs().max()
