"""Launches of the single-launch and batched solvers: repeated, from other streams, beside other work."""

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
