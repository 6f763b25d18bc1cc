"""P2 plans whose solver rows are ordered by edge class (``femk_order.cu``) against the canonical CSR.

The solvers' operator holds the CSR's values in another row order, with column tables of up to four runs of rows a
slice. ``solver_layout`` = 0 keeps the CSR: two CG steps from the same start differ by the rounding of the row sums
and dot products alone (rows of up to 65 entries: below 65 eps of |A| |x| each, amplified by the two quotients; 1e-11
of the largest entry holds with room), whole solves by the stop rule, 1e-7 as elsewhere."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import mesh as om  # noqa: E402

# (dim, cells per axis): lines longer and shorter than a slice (P2 lines of 2 rows up: more runs than a table holds),
# below and above the 65,536 unknowns from which tables are built, one cell a side
BOXES = [
    (3, (20, 21, 22)),
    (3, (13, 90, 9)),
    (3, (160, 40, 2)),
    (3, (9, 4, 260)),
    (3, (6, 5, 7)),
    (3, (1, 1, 1)),
    (2, (150, 120)),
    (2, (3000, 6)),
    (2, (6, 3000)),
    (2, (11, 13)),
]


def _mesh(dim, n, seed=7):
    from jno_b200.domain import box_points_tets, jitter_interior, jitter_interior_2d, rect_points_tris

    if dim == 3:
        pts, cells = box_points_tets(*n)
        return jitter_interior(pts, *n, seed=seed), cells
    pts, cells = rect_points_tris(*n)
    return jitter_interior_2d(pts, *n, seed=seed)[:, :2], cells


@pytest.mark.parametrize("dim,n", BOXES)
def test_products_and_steps_match_the_csr(dim, n):
    from jno_b200.plan import FemPlan

    pts, cells = _mesh(dim, n)
    plan, csr = FemPlan(pts, cells, 2, options={"ring64": 14}), FemPlan(pts, cells, 2, options={"solver_layout": 0})
    logk = torch.as_tensor(om.logk_field(len(cells), 1017), device="cuda")
    vals, b = plan.assemble(logk, g=torch.linspace(0.0, 1.0, plan.n, dtype=torch.float64, device="cuda"))
    inv = plan.jacobi(vals)
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(plan.n, dtype=torch.float64, device="cuda", generator=g)
    plan.prepare_operator(vals)
    y, z = plan.spmv_prepared(x), plan.spmv(vals, x)
    assert (y - z).abs().max() <= 65 * 2.3e-16 * plan.spmv(vals.abs(), x.abs()).abs().max()
    for steps in (1, 2):
        u, v = (p.pcg(vals, b, x.clone(), inv, 1e-14, maxiter=steps)[0] for p in (plan, csr))
        assert (u - v).abs().max() <= 1e-11 * max(1.0, v.abs().max().item())
    for solve in ("pcg", "mixed", "bicgstab", "gmres"):
        got = []
        for p in (plan, csr):
            if solve == "pcg":
                got.append(p.pcg(vals, b, x.clone(), inv, 1e-10)[0])
            elif solve == "mixed" and max(n) < 1000:
                # (FP32 steps and BiCGStab do not converge on the 500:1 boxes, whatever the layout)
                u, _, _, _, st = p.pcg_mixed(vals, b, inv, None, 1e-10)
                assert st == 0
                got.append(u)
            elif solve == "bicgstab" and p is plan and max(n) < 1000:
                u, _, _, st = p.bicgstab(vals, b, x.clone(), inv, 1e-11)
                assert st == 0
                got.append(u)
            elif solve == "gmres" and plan.n < 3000:
                got.append(p.gmres(vals, b, None, inv, 1e-10, restart=40)[0])
        if solve == "bicgstab" and got:
            got.append(csr.pcg(vals, b, x.clone(), inv, 1e-11)[0])  # the CSR layout has no BiCGStab
        if got:
            assert (torch.linalg.norm(got[0] - got[1]) / torch.linalg.norm(got[1])).item() <= 1e-7, solve


def test_batched_solves_put_a_plan_back_into_the_dof_order():
    """The batched solvers' problems own runs of DOFs: on a P2 plan with its own row order they rebuild the solver's
    operator in the DOF order, and the other solvers go on with that."""
    from jno_b200.plan import FemPlan

    pts, cells = _mesh(3, (5, 6, 4))
    plan = FemPlan(pts, cells, 2)
    logk = torch.as_tensor(om.logk_field(len(cells), 1018), device="cuda")
    vals, b = plan.assemble(logk)
    inv = plan.jacobi(vals)
    before = plan.pcg(vals, b, None, inv, 1e-10)[0]
    x, it, rel, stv, st = plan.pcg_batched([0, plan.n], vals, b, None, inv, 1e-10)
    after = plan.pcg(vals, b, None, inv, 1e-10)[0]
    mixed = plan.pcg_mixed(vals, b, inv, None, 1e-10)[0]
    assert st == 0
    for u in (x, after, mixed):
        assert (torch.linalg.norm(u - before) / torch.linalg.norm(before)).item() <= 1e-7


def test_prepared_products_are_capturable_and_hold_no_state():
    """``spmv_prepared`` on a plan with a row order, straight after ``prepare_operator``: captured in a CUDA graph, and
    on two streams at once, the bits of the plain call."""
    from jno_b200.plan import FemPlan

    pts, cells = _mesh(3, (14, 11, 12))
    plan = FemPlan(pts, cells, 2)
    vals, _ = plan.assemble(torch.as_tensor(om.logk_field(len(cells), 1020), device="cuda"))
    plan.prepare_operator(vals)
    g = torch.Generator(device="cuda").manual_seed(3)
    xs = [torch.randn(plan.n, dtype=torch.float64, device="cuda", generator=g) for _ in range(2)]
    ys = [torch.zeros_like(x) for x in xs]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.spmv_prepared(xs[0], ys[0])
    graph.replay()
    torch.cuda.synchronize()
    want = [plan.spmv_prepared(x) for x in xs]
    assert torch.equal(ys[0], want[0])
    streams = [torch.cuda.Stream() for _ in xs]
    torch.cuda.synchronize()
    for _ in range(20):
        for s, x, y in zip(streams, xs, ys):
            with torch.cuda.stream(s):
                plan.spmv_prepared(x, y)
    torch.cuda.synchronize()
    assert torch.equal(ys[0], want[0]) and torch.equal(ys[1], want[1])
