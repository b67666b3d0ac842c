"""Batched Standard cycles whose members' coarse levels take different forms of the level product: a member whose
level 1 (30,625 nodes) is above the split form's limit next to one below it.  The batch launches each form for its own
members (so one kernel more per product than a batch of the large member alone, whose other levels are small), and both
members equal their solo runs bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REGIME = dict(oc_sum_order=1, mg_coarse_assembly=1, mg_vcycle=1, mg_rebuild_period=1, cg_tol=1e-6, cg_max_it=2000)
LARGE, SMALL = (96, 192, 96), (16, 48, 24)


def test_members_on_both_sides_of_the_split_limit():
    import algorithmengineering_altproject_b200 as t3d
    B = t3d.Batch([LARGE], **REGIME)
    alone = B.info()["kernels_per_iteration"]
    B.close()
    dims = [SMALL, LARGE]
    B = t3d.Batch(dims, **REGIME)
    assert B.info()["kernels_per_iteration"] == alone + 2   # level 1 down and up
    V0 = [0.2, 0.12]
    cs = B.design_init(V0)
    recs = B.run([2, 2])
    xs = [m.density() for m in B.members]
    us = [m.displacement() for m in B.members]
    B.close()
    for i, d in enumerate(dims):
        P = t3d.Problem(*d, precision=t3d.T3D_MIXED, matvec32_tile=t3d.T3D_BATCH_TILE, **REGIME)
        assert P.design_init(V0[i]) == cs[i]
        for k in range(2):
            r = P.design_step()
            assert (r["obj"], r["pcg_iters"]) == (recs[i][k]["obj"], recs[i][k]["pcg_iters"])
        np.testing.assert_array_equal(P.density(), xs[i])
        np.testing.assert_array_equal(P.displacement(), us[i])
        P.close()
