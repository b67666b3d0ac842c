"""A context holds all its device memory from creation on: a finished design can be read back, and the serving loop's
footprint per node, learned at creation, covers a request's whole life."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [dict(), dict(oc_sum_order=1), dict(oc_sum_order=1, precision=1, mg_vcycle=1)])
@pytest.mark.parametrize("voids", [(), ((30.0, 10.0, 12.0, 9.0, 5.0, 5.0),)])
def test_no_device_memory_after_creation(kw, voids):
    import algorithmengineering_altproject_b200 as t3d
    P = t3d.Problem(20, 61, 23, problem=t3d.ProblemSpec.make(0, voids), cg_max_it=30, **kw)
    held = P.device_bytes
    assert P.info().device_bytes == held
    P.design_init(0.2)
    P.design_step()
    x, u = P.density(), P.displacement()
    assert x.size == P.ne and u.size == P.nf == P.free_dofs().size
    y = P.K_times_u_finest(P.simp(x), u)
    P.oc_update(x, -np.ones(P.ne, np.float32), 0.2)
    assert np.all(np.isfinite(y)) and P.info().device_bytes == held
    P.close()
