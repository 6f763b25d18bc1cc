"""The matrix-free CG step (product with its share of <p, A p>, fused vector kernels, replayed as a graph) against
the assembled operator's CG: the same system, so the solutions agree to the stop rule (1e-10 here; 1e-7 of the
solution with condition numbers below 1e3, as elsewhere)."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import mesh as om  # noqa: E402


def _mesh(dim, n, shuffled, seed=9):
    from jno_b200.domain import box_points_tets, jitter_interior, jitter_interior_2d, rect_points_tris

    if dim == 3:
        pts, cells = box_points_tets(*n)
        pts = jitter_interior(pts, *n, seed=seed)
    else:
        pts, cells = rect_points_tris(*n)
        pts = jitter_interior_2d(pts, *n, seed=seed)[:, :2]
    if shuffled:
        cells = cells[np.random.default_rng(seed).permutation(len(cells))]
    return pts, cells


@pytest.mark.parametrize("dim,n,order,shuffled", [(3, (11, 9, 10), 1, False), (3, (1, 1, 1), 1, False),
                                                  (3, (11, 9, 10), 1, True), (3, (4, 5, 6), 2, False),
                                                  (2, (17, 14), 1, False), (2, (9, 8), 2, True)])
@pytest.mark.parametrize("precond", [True, False])
def test_matrix_free_cg_matches_the_assembled_one(dim, n, order, shuffled, precond):
    from jno_b200.plan import FemPlan

    pts, cells = _mesh(dim, n, shuffled)
    plan = FemPlan(pts, cells, order)
    g = torch.linspace(-1.0, 1.0, plan.n, dtype=torch.float64, device="cuda")
    for field, scale in ((1019, 1.0), (1020, 2.5)):  # another coefficient and scale: another captured step
        logk = torch.as_tensor(om.logk_field(len(cells), field), device="cuda")
        vals, b = plan.assemble(logk, scale=scale, g=g)
        inv = plan.jacobi(vals) if precond else None
        ref = plan.pcg(vals, b, None, inv, 1e-10)[0]
        for shift in (0, 1):  # an 8-byte offset runs the vector kernels of unaligned callers
            x = torch.zeros(plan.n + 1, dtype=torch.float64, device="cuda")[shift: shift + plan.n]
            for _ in range(2):  # the second solve starts from the solution
                _, it, rel, st = plan.pcg_matfree(logk, b, x, inv, scale=scale, tol=1e-10)
                assert st == 0 and rel <= 2e-10
                assert (torch.linalg.norm(x - ref) / torch.linalg.norm(ref)).item() <= 1e-7
            assert it <= 1


def test_matrix_free_status_paths():
    from jno_b200 import _lib
    from jno_b200.plan import FemPlan

    pts, cells = _mesh(3, (7, 6, 8), False)
    plan = FemPlan(pts, cells, 1)
    logk = torch.as_tensor(om.logk_field(len(cells), 1021), device="cuda")
    vals, b = plan.assemble(logk)
    inv = plan.jacobi(vals)
    for maxiter in (0, 1, 5):
        x, it, rel, st = plan.pcg_matfree(logk, b, None, inv, tol=1e-12, maxiter=maxiter)
        y, ity, _, sty = plan.pcg(vals, b, None, inv, 1e-12, maxiter=maxiter)
        assert (it, st) == (ity, sty) == (maxiter, _lib.FEMK_NOT_CONVERGED)
        assert (x - y).abs().max() <= 1e-11 * max(1e-300, y.abs().max().item())
    with pytest.raises(_lib.FemkError, match="positive definite"):
        plan.pcg_matfree(logk, b, None, inv, scale=-1.0)
    bad = b.clone()
    bad[plan.n // 2] = float("nan")
    with pytest.raises(_lib.FemkError, match="non-finite"):
        plan.pcg_matfree(logk, bad, None, inv)
    assert plan.pcg_matfree(logk, b, None, inv)[3] == 0
