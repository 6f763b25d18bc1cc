"""P1 plans whose solver reads its columns from tables by runs of rows (``femk_order.cu``) against the canonical CSR.

Products: rows of up to 15 entries (lattices; irregular rows below 40) summed in another order, below 40 eps of the
largest |A| |x|. Two CG steps from the same start: rounding of the row sums and dot products amplified by the two
quotients, 1e-11 of the largest entry holds with room. Solves by the stop rule, 1e-7 as elsewhere."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import mesh as om  # noqa: E402

# (dim, cells per axis, shuffled numbering): lines longer and shorter than a slice (up to 16 runs a slice: past what a
# table holds), lines of just a slice (one run a slice and its ends), one cell, and no lines at all
BOXES = [
    (3, (31, 30, 29), False),
    (3, (40, 41, 42), False),
    (3, (2, 150, 160), False),
    (3, (160, 150, 2), False),
    (3, (5, 70, 6), False),
    (3, (1, 1, 1), False),
    (3, (40, 41, 42), True),
    (2, (300, 280), False),
    (2, (3, 9000), False),
    (2, (9000, 3), False),
    (2, (31, 4), False),
]


@pytest.mark.parametrize("bulk", [False, True])
@pytest.mark.parametrize("dim,n,shuffled", BOXES)
def test_products_and_steps_match_the_csr(dim, n, shuffled, bulk):
    from jno_b200.domain import box_points_tets, jitter_interior, jitter_interior_2d, rect_points_tris
    from jno_b200.plan import FemPlan

    if dim == 3:
        pts, cells = box_points_tets(*n)
        pts = jitter_interior(pts, *n, seed=9)
    else:
        pts, cells = rect_points_tris(*n)
        pts = jitter_interior_2d(pts, *n, seed=9)[:, :2]
    if shuffled:
        to = np.random.default_rng(4).permutation(len(pts))
        moved = np.empty_like(pts)
        moved[to] = pts
        pts, cells = moved, to[cells].astype(cells.dtype)
    plan = FemPlan(pts, cells, 1, options={"ring64": 14} if bulk else None)
    csr = FemPlan(pts, cells, 1, options={"solver_layout": 0})
    logk = torch.as_tensor(om.logk_field(len(cells), 1019), device="cuda")
    vals, b = plan.assemble(logk, g=torch.linspace(0.0, 1.0, plan.n, dtype=torch.float64, device="cuda"))
    inv = plan.jacobi(vals)
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(plan.n, dtype=torch.float64, device="cuda", generator=g)
    plan.prepare_operator(vals)
    y, z = plan.spmv_prepared(x), plan.spmv(vals, x)
    assert (y - z).abs().max() <= 40 * 2.3e-16 * plan.spmv(vals.abs(), x.abs()).abs().max()
    for steps in (1, 2):
        u, v = (p.pcg(vals, b, x.clone(), inv, 1e-14, maxiter=steps)[0] for p in (plan, csr))
        assert (u - v).abs().max() <= 1e-11 * max(1.0, v.abs().max().item())
    if max(n) < 1000:
        u, v = (p.pcg(vals, b, None, inv, 1e-10)[0] for p in (plan, csr))
        assert (torch.linalg.norm(u - v) / torch.linalg.norm(v)).item() <= 1e-7
        u, _, _, _, st = plan.pcg_mixed(vals, b, inv, None, 1e-10)
        assert st == 0 and (torch.linalg.norm(u - v) / torch.linalg.norm(v)).item() <= 1e-7
