"""Batched PCG with a set of blocks a problem (``femk_batch_sets.cu``) against the grid form and the single solver.

``ring64`` = 14 selects the kernels of the chunked solvers, and with them the grid form, which takes the same steps and
sums in another order: the solutions of both meet a stop rule of 1e-10 (cond * tol well below 1e-7, the bound of the
other batched tests), and the step counts differ by at most one."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import mesh as om  # noqa: E402

# sides of a batch's cubes: a block each; clusters of 2 .. 16; the grid's groups, alone, beside clusters, in two
# launches of different groups, and more problems than groups; more problems than sets
BATCHES = [
    [1, 2, 3, 9, 10, 11],
    [4] * 200,
    [12, 20, 13, 17],
    [25, 5, 31, 11, 22, 3],
    [40, 41, 9],
    [34],
    [48, 3, 12],
    [46, 2, 47, 30, 48],
    [56, 30, 30, 30, 31, 32, 33, 29, 28],
]


def _problems(sides):
    out = []
    for i, n in enumerate(sides):
        pts, tets = om.equi_distant_box(n, n, n)
        out.append((om.jitter_interior(pts, n, n, n, seed=70 + i), tets))
    return out, [om.logk_field(len(t), 900 + i) for i, (_, t) in enumerate(out)]


@pytest.mark.parametrize("sides", BATCHES, ids=lambda s: f"{len(s)}x{max(s)}")
def test_sets_match_the_grid_form(sides):
    from jno_b200.batch import BatchedPoisson

    meshes, logk = _problems(sides)
    got = []
    for opts in ({}, {"ring64": 14}):
        batch = BatchedPoisson(meshes, options=opts or None)
        vals, b = batch.assemble(logk)
        inv = batch.plan.jacobi(vals)
        g = torch.Generator(device="cuda").manual_seed(2)
        x0 = torch.randn(batch.plan.n, dtype=torch.float64, device="cuda", generator=g) * (b != 0)
        for dinv, start in ((inv, None), (None, None), (inv, x0)):
            got.append(batch.plan.pcg_batched(batch.row_off, vals, b, None if start is None else start.clone(), dinv,
                                              1e-10, 0.0, 20_000, 64, 2))
        got.append(batch.plan.pcg_batched(batch.row_off, vals, b, None, inv, 1e-10, 0.0, 5, 64, 2))
        row_off = batch.row_off
    for k in range(4):
        (x, it, rel, stv, st), (y, jt, sel, ttv, tt) = got[k], got[k + 4]
        assert st == tt and np.array_equal(stv, ttv)
        if k == 3:
            assert np.array_equal(it, jt)  # the cap, or problems that need fewer steps
            assert (x - y).abs().max() <= 1e-9 * y.abs().max()
            continue
        if k == 0:
            assert np.abs(np.asarray(it) - np.asarray(jt)).max() <= 1
            assert np.all(np.asarray(rel)[np.asarray(it) > 0] <= 2e-10)
        for i in range(len(sides)):
            u, v = x[row_off[i]:row_off[i + 1]], y[row_off[i]:row_off[i + 1]]
            assert torch.linalg.norm(u - v) <= 1e-7 * torch.linalg.norm(v)


@pytest.mark.parametrize("sides", [[6, 9, 5], [48, 40, 12]])
def test_problems_that_fail_do_so_alone(sides):
    """A negative definite problem breaks down, one with a NaN in its load says so; the others solve."""
    from jno_b200 import _lib
    from jno_b200.batch import BatchedPoisson

    meshes, logk = _problems(sides)
    batch = BatchedPoisson(meshes)
    vals, b = batch.assemble(logk)
    off = batch.row_off
    ptr = batch.plan.pattern()[0]
    inv = batch.plan.jacobi(vals)
    bad = vals.clone()
    bad[int(ptr[int(off[1])]):int(ptr[int(off[2])])] *= -1.0
    load = b.clone()
    load[int(off[2]) + 3] = float("nan")
    x = torch.zeros_like(b)
    with pytest.raises(_lib.FemkError) as err:
        batch.plan.pcg_batched(off, bad, load, x, inv, 1e-10, 0.0, 1000, 64, 2)
    assert err.value.status == _lib.FEMK_NONFINITE  # the last problem's
    y = batch.plan.pcg_batched(off, vals, b, None, inv, 1e-10, 0.0, 1000, 64, 2)[0]
    n = int(off[1])
    assert torch.linalg.norm(x[:n] - y[:n]) <= 1e-7 * torch.linalg.norm(y[:n])


@pytest.mark.parametrize("order,n,shuffled", [(1, 33, True), (1, 9, True), (2, 20, False), (2, 7, True)])
def test_one_problem_is_the_single_solve(order, n, shuffled):
    """P2 rows and numberings without tables (other column types) as a batch of one."""
    from jno_b200.plan import FemPlan

    pts, cells = om.equi_distant_box(n, n, n)
    if shuffled:
        to = np.random.default_rng(4).permutation(len(pts))
        moved = np.empty_like(pts)
        moved[to] = pts
        pts, cells = moved, to[cells].astype(cells.dtype)
    plan = FemPlan(pts, cells, order)
    vals, b = plan.assemble(torch.as_tensor(om.logk_field(len(cells), 77), device="cuda"))
    inv = plan.jacobi(vals)
    x = plan.pcg_batched([0, plan.n], vals, b, None, inv, 1e-10)[0]
    y = plan.pcg(vals, b, None, inv, 1e-10)[0]
    assert torch.linalg.norm(x - y) <= 1e-7 * torch.linalg.norm(y)


def test_the_tuner_times_the_form_that_has_a_schedule(monkeypatch):
    """FP64 batches that run a problem at a time have no schedule: the candidates are timed on the mixed solve; with the
    grid form's kernels selected, on the FP64 solve."""
    from jno_b200 import tuner
    from jno_b200.batch import BatchedPoisson

    meshes, logk = _problems([6, 9, 5])
    for opts, called in ((None, "pcg_batched_mixed"), ({"ring64": 14}, "pcg_batched")):
        batch = BatchedPoisson(meshes, options=opts)
        vals, b = batch.assemble(logk)
        inv = batch.plan.jacobi(vals)
        calls = []
        for name in ("pcg_batched", "pcg_batched_mixed"):
            def wrap(*a, _f=getattr(batch.plan, name), _n=name):
                calls.append(_n)
                return _f(*a)
            monkeypatch.setattr(batch.plan, name, wrap)
        best, times = tuner.tune(batch, vals, b, inv, 1e-8, [(64, 1), (128, 2)], reps=1)
        assert set(calls[1:]) == {called} and len(calls) == 6 and len(times) == 2
