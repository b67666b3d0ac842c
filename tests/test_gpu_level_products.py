"""The Standard V-cycle's coarse-level products on both sides of the level size at which they change form (one block
per 32 nodes with the elements split over its warps; a thread per node), with level sizes that divide no block:
the FP64 cycle is symmetric, and the FP32 cycle -- packed matrices, three rows a thread -- agrees with it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(8, 40, 24), (33, 57, 41), (80, 176, 96), (96, 192, 96)])
def test_coarse_level_products(dims):
    import algorithmengineering_altproject_b200 as t3d
    P = t3d.Problem(*dims, mg_vcycle=t3d.T3D_VCYCLE_STANDARD, precision=t3d.T3D_MIXED)
    rng = np.random.default_rng(3)
    P.make_diagonal_preconditioner_from_static(1e-3 + rng.random(P.ne) ** 3)
    a, b = (rng.standard_normal(P.nf).astype(np.float32).astype(np.float64) for _ in range(2))
    za, zb = P.vcycle(a), P.vcycle(b)
    assert abs(a @ zb - b @ za) <= 1e-10 * np.linalg.norm(a) * np.linalg.norm(zb)
    assert a @ za > 0 and b @ zb > 0
    z32 = P.vcycle32(a)
    assert np.linalg.norm(z32 - za) <= 1e-5 * np.linalg.norm(za)
    P.close()
