"""Launches of the single-launch and batched solvers: which systems take them, repeated, from other streams, beside
other work."""

import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import mesh as om  # noqa: E402


def _plan(n, order=1, options=None):
    from jno_b200.plan import FemPlan

    pts, cells = om.equi_distant_box(*n)
    return FemPlan(pts, cells, order, options=options), torch.as_tensor(om.logk_field(len(cells), 1021), device="cuda")


@pytest.mark.parametrize("n", [(9, 10, 11), (10, 11, 13), (15, 16, 17), (24, 25, 23)])
def test_cluster_launches_repeat_to_the_bit(n):
    """Clusters of 2, 4, 8 and 16 blocks launched one after another: their sums go through each other's shared memory,
    and a store that a block of the cluster did not get would show in the bits."""
    plan, logk = _plan(n)
    vals, b = plan.assemble(logk)
    inv = plan.jacobi(vals)
    want = plan.pcg(vals, b, None, inv, 1e-10), plan.bicgstab(vals, b, None, inv, 1e-10)
    for _ in range(100):
        got = plan.pcg(vals, b, None, inv, 1e-10), plan.bicgstab(vals, b, None, inv, 1e-10)
        for w, g in zip(want, got):
            assert torch.equal(w[0], g[0]) and w[1:] == g[1:]


def test_batches_on_clusters_repeat_to_the_bit():
    from jno_b200.batch import BatchedPoisson

    meshes = [om.equi_distant_box(n, n, n) for n in (12, 13, 16, 20, 25) * 8]
    batch = BatchedPoisson(meshes)
    vals, b = batch.assemble([om.logk_field(len(t), 930 + i) for i, (_, t) in enumerate(meshes)])
    inv = batch.plan.jacobi(vals)
    x, it = batch.plan.pcg_batched(batch.row_off, vals, b, None, inv, 1e-10)[:2]
    for _ in range(30):
        y, jt = batch.plan.pcg_batched(batch.row_off, vals, b, None, inv, 1e-10)[:2]
        assert torch.equal(x, y) and np.array_equal(it, jt)


# (dim, cells per axis, order, shuffled, CG in one launch, BiCGStab in one launch): either side of what stays on the
# chip, where a row has few entries (so that the vectors count) and many, with and without shared columns
LARGE = [
    (2, (850, 850), 1, False, True, True),
    (2, (960, 960), 1, False, False, False),
    (3, (86, 86, 86), 1, False, True, False),
    (3, (88, 88, 88), 1, False, False, False),
    (2, (400, 400), 2, False, True, True),
    (2, (445, 445), 2, False, False, False),
    (3, (35, 35, 35), 2, False, True, True),
    (2, (300, 300), 2, True, True, True),
    (2, (370, 370), 2, True, False, False),
    (2, (800, 800), 1, True, True, False),
]


@pytest.mark.parametrize("dim,n,order,shuffled,cg,bicg", LARGE)
def test_systems_past_the_chip_keep_the_chunked_solvers(dim, n, order, shuffled, cg, bicg):
    """Few launches tell the single launch. Its first two iterates agree with the chunked solver's to the rounding of
    row sums, dot products and two quotients: 1e-11 of the largest entry holds with room."""
    from jno_b200 import _lib
    from jno_b200.domain import box_points_tets, rect_points_tris
    from jno_b200.plan import FemPlan

    pts, cells = box_points_tets(*n) if dim == 3 else rect_points_tris(*n)
    pts = pts[:, :dim]
    if shuffled:
        to = np.random.default_rng(4).permutation(len(pts))
        moved = np.empty_like(pts)
        moved[to] = pts
        pts, cells = moved, to[cells]
    plan = FemPlan(pts, cells, order)
    chunked = FemPlan(pts, cells, order, options={"ring64": 14})
    vals, b = plan.assemble(torch.zeros(len(cells), dtype=torch.float64, device="cuda"))
    inv = plan.jacobi(vals)
    b = torch.randn(plan.n, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(6))
    launches = _lib.load().femk_kernel_launches
    for name, one in (("pcg", cg), ("bicgstab", bicg)):
        before = launches()
        getattr(plan, name)(vals, b, None, inv, 1e-14, maxiter=30)
        assert (launches() - before <= 5) == one, name
        x, y = (getattr(p, name)(vals, b, None, inv, 1e-14, maxiter=2)[0] for p in (plan, chunked))
        assert (x - y).abs().max() <= 1e-11 * y.abs().max()


def _shuffled(pts, cells, seed):
    to = np.random.default_rng(seed).permutation(len(pts))
    moved = np.empty_like(pts)
    moved[to] = pts
    return moved, to[cells]


# (side, problems, numbering, the grid form): thousands of tiny problems, and neighbouring rows whose columns lie apart,
# where the grid form is the faster one
FORMS = [
    (3, 500, "lattice", False),
    (3, 7000, "lattice", True),
    (1, 3500, "lattice", True),
    (5, 3500, "lattice", False),
    (30, 10, "lattice", False),
    (30, 10, "shuffled", True),
    (30, 5, "shuffled", False),
    (12, 120, "shuffled", False),
]


@pytest.mark.parametrize("side,count,numbering,grid", FORMS)
def test_batches_take_the_form_that_is_faster(side, count, numbering, grid):
    """Whichever form a batch takes, its solutions are those of the grid form (the bounds of the other batched tests)."""
    from jno_b200.batch import BatchedPoisson

    mesh = om.equi_distant_box(side, side, side)
    if numbering == "shuffled":
        mesh = _shuffled(*mesh, 3)
    got = []
    for opts in (None, {"ring64": 14}):
        batch = BatchedPoisson([mesh] * count, options=opts)
        logk = torch.as_tensor(om.logk_field(batch.plan.ntet, 941), device="cuda")
        vals, b = batch.plan.assemble(logk)
        x, it = batch.plan.pcg_batched(batch.row_off, vals, b, None, batch.plan.jacobi(vals), 1e-10)[:2]
        got.append((x.view(count, -1), np.asarray(it)))
        assert batch.plan.batch_graph == (grid or opts is not None)
    (x, it), (y, jt) = got
    assert np.abs(it - jt).max() <= 1
    assert torch.all(torch.linalg.norm(x - y, dim=1) <= 1e-7 * torch.linalg.norm(y, dim=1))


@pytest.mark.parametrize("n", [(33, 35, 31), (10, 11, 13)])
@pytest.mark.parametrize("solver", ["pcg", "bicgstab", "pcg_mixed"])
def test_the_first_solve_of_a_plan_on_a_side_stream_beside_a_busy_default_stream(n, solver):
    """A plan's workspaces are made during its first solve. Whatever clears them is in the solve's own stream: the
    default stream's pending work (a sleeping kernel) delays nothing and the second solve has the same bits."""
    from jno_b200.plan import FemPlan

    pts, cells = om.equi_distant_box(*n)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)  # about 0.1 s of one thread
    with torch.cuda.stream(side):
        plan = FemPlan(pts, cells, 1)
        vals, b = plan.assemble(torch.zeros(len(cells), dtype=torch.float64, device="cuda"))
        inv = plan.jacobi(vals)
        args = (vals, b, inv, None, 1e-10) if solver == "pcg_mixed" else (vals, b, None, inv, 1e-10)
        got = [getattr(plan, solver)(*args) for _ in range(2)]
    torch.cuda.synchronize()
    assert got[0][-1] == 0 and got[0][1:] == got[1][1:] and torch.equal(got[0][0], got[1][0])
    assert (torch.linalg.norm(b - plan.spmv(vals, got[0][0])) <= 2e-10 * torch.linalg.norm(b)).item()


@pytest.mark.parametrize("mixed", [False, True])
def test_batched_calls_leave_a_plan_s_own_row_order(mixed):
    """A P2 lattice plan solves in a row order of its own, batches in the DOF order. Neither a batched call that is
    refused nor one that runs changes what the plan's other calls do: to the bit, prepared operator included."""
    from jno_b200 import _lib

    plan, logk = _plan((9, 8, 10), 2)
    vals, b = plan.assemble(logk)
    inv = plan.jacobi(vals)
    info = _lib.PlanInfo()

    def layout():
        _lib.check(plan._lib.femk_plan_get_info(plan.handle, ctypes.byref(info)))
        return info.sell_nnz, info.sell_col_units

    def calls():
        return (plan.pcg(vals, b, None, inv, 1e-10)[:3], plan.bicgstab(vals, b, None, inv, 1e-10)[:3],
                plan.pcg_mixed(vals, b, inv, None, 1e-8)[:4])

    def batched(off):
        if mixed:
            return plan.pcg_batched_mixed(off, vals, b, inv, None, 1e-8)
        return plan.pcg_batched(off, vals, b, None, inv, 1e-10)

    before, want = layout(), calls()
    x = torch.randn(plan.n, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    plan.prepare_operator(vals)
    y = plan.spmv_prepared(x)
    for off in ([0, plan.n - 1], [0, 7, 7, plan.n], [1, plan.n]):
        with pytest.raises(_lib.FemkError):
            batched(off)
        assert layout() == before and torch.equal(plan.spmv_prepared(x), y)
    for _ in range(2):
        u = batched([0, plan.n])[0]
        assert (torch.linalg.norm(u - want[0][0]) <= 1e-6 * torch.linalg.norm(u)).item()
        assert layout() == before and torch.equal(plan.spmv_prepared(x), y)
        for w, g in zip(want, calls()):
            assert torch.equal(w[0], g[0]) and w[1:] == g[1:]
        plan.prepare_operator(vals)


@pytest.mark.parametrize("spokes", [200, 253, 254, 300, 500, 1200])
def test_rows_of_255_entries_are_refused_as_such(spokes):
    """A vertex that all triangles share: 254 entries a row are the most, and more are an argument error with that
    message, however many."""
    from scipy.sparse import csr_matrix

    from jno_b200 import _lib
    from jno_b200.plan import FemPlan

    turn = 2.0 * np.pi * np.arange(spokes) / spokes
    pts = np.concatenate([[[0.0, 0.0]], np.stack([np.cos(turn), np.sin(turn)], 1)])
    rim = 1 + np.arange(spokes)
    cells = np.stack([np.zeros_like(rim), rim, np.roll(rim, -1)], 1)
    if spokes >= 254:
        with pytest.raises(_lib.FemkError, match="255 or more entries") as err:
            FemPlan(pts, cells, 1)
        assert err.value.status == _lib.FEMK_EINVAL
        return
    plan = FemPlan(pts, cells, 1)
    vals, b = plan.assemble(torch.zeros(spokes, dtype=torch.float64, device="cuda"))
    x = np.random.default_rng(1).normal(size=plan.n)
    ptr, col = (t.cpu().numpy() for t in plan.pattern())
    want = csr_matrix((vals.cpu().numpy(), col, ptr), shape=(plan.n, plan.n)) @ x
    got = plan.spmv(vals, torch.as_tensor(x, device="cuda")).cpu().numpy()
    assert np.abs(got - want).max() <= 1e-14 * spokes * np.abs(vals.cpu().numpy()).max() * np.abs(x).max()


def test_solves_of_two_plans_at_once_have_the_bits_of_one_alone():
    """Two threads, a stream and a plan each: launches that want every SM (a grid of all blocks, a cluster, a batch)
    take turns or share the device, and neither runs out of time nor changes the other's result."""
    import threading

    from jno_b200.batch import BatchedPoisson

    def prepare(n):
        plan, logk = _plan(n)
        vals, b = plan.assemble(logk)
        inv = plan.jacobi(vals)
        return [lambda: plan.pcg(vals, b, None, inv, 1e-10)[:3], lambda: plan.bicgstab(vals, b, None, inv, 1e-10)[:3]]

    meshes = [om.equi_distant_box(n, n, n) for n in (40, 12, 14, 20)]
    batch = BatchedPoisson(meshes)
    bvals, load = batch.assemble([om.logk_field(len(t), 950 + i) for i, (_, t) in enumerate(meshes)])
    binv = batch.plan.jacobi(bvals)
    calls = [*prepare((45, 46, 47)), *prepare((24, 25, 23)), *prepare((33, 35, 31)),
             lambda: batch.plan.pcg_batched(batch.row_off, bvals, load, None, binv, 1e-10)[:1]]
    split = calls[:2] + calls[6:], calls[2:6]
    torch.cuda.synchronize()
    want = [[f() for f in mine] for mine in split]
    got, failed = [[], []], []

    def run(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(20):
                    got[k].append([f() for f in split[k]])
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001 - reported by the test's thread
            failed.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=run, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for k in range(2):
        assert len(got[k]) == 20
        for results in got[k]:
            for w, g in zip(want[k], results):
                assert torch.equal(w[0], g[0]) and w[1:] == g[1:]


def test_a_batch_group_s_wait_that_runs_out_is_a_status():
    """Block 0 of the group that solves the one problem never arrives: the others give up after the limit, the call
    reports it and leaves the problem that status, and the device goes on."""
    from jno_b200 import _lib

    bad, logk = _plan((34, 33, 32), options={"test_skip_arrival": 0, "barrier_limit_ms": 5.0})
    vals, b = bad.assemble(logk)
    inv = bad.jacobi(vals)
    for _ in range(2):
        status = np.zeros(1, dtype=np.int32)
        off = np.asarray([0, bad.n], dtype=np.int64)
        x = torch.zeros_like(b)
        st = bad._lib.femk_pcg_batched(bad.handle, 1, ctypes.c_void_p(off.ctypes.data), _lib.ptr(vals), _lib.ptr(b),
                                       _lib.ptr(x), _lib.ptr(inv), 1e-8, 0.0, 1000, 64, 2, None, None,
                                       ctypes.c_void_p(status.ctypes.data), _lib.stream_handle())
        assert st == _lib.FEMK_TIMEOUT and status[0] == _lib.FEMK_TIMEOUT
        assert b"gave up" in bad._lib.femk_last_error_string()
    good = _plan((34, 33, 32))[0]
    x, it, rel, stv, st = good.pcg_batched([0, good.n], vals, b, None, inv, 1e-8)
    assert st == 0 and rel[0] <= 2e-8 and not good.batch_graph
