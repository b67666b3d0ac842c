"""The Adapted V-cycle's forms for a level 1 of more than 100,000 nodes -- the first restriction in one pass per axis,
a node's three components in one thread of the level's prolongation -- against the oracle, bit for bit, on a grid of
ragged sides (level 1 has 77 x 37 x 39 nodes); and the FP32 cycle's restriction at that size against the FP64 cycle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_adapted_vcycle_large_level_bit_exact_with_oracle():
    import algorithmengineering_altproject_b200 as t3d
    from oracle.bindings import Oracle
    dims = (143, 301, 150)
    P = t3d.Problem(*dims)
    O = Oracle(*dims, red_mode=1, pow_mode=0, vol_mode=0, approx_mode=0)
    rng = np.random.default_rng(23)
    E = np.where(rng.random(P.ne) < 0.3, 1e-6, rng.uniform(0.05, 1.0, P.ne))
    P.make_diagonal_preconditioner_from_static(E)
    O.mg_build(E)
    r = rng.standard_normal(P.nf)
    n0 = P.kernel_launches()
    z = P.vcycle(r)
    # x, y and z passes, a kernel per further restriction, the coarsest solve, a prolongation per transition
    L = len(P.levels)
    assert P.kernel_launches() - n0 == 3 + (L - 2) + 1 + (L - 1)
    np.testing.assert_array_equal(z, O.vcycle(r))
    P.close()


def test_fp32_adapted_vcycle_large_level_matches_fp64():
    import algorithmengineering_altproject_b200 as t3d
    P = t3d.Problem(143, 301, 150, precision=t3d.T3D_MIXED)
    rng = np.random.default_rng(29)
    P.make_diagonal_preconditioner_from_static(rng.uniform(0.05, 1.0, P.ne))
    r = rng.standard_normal(P.nf).astype(np.float32).astype(np.float64)
    z = P.vcycle(r)
    assert np.linalg.norm(P.vcycle32(r) - z) <= 1e-5 * np.linalg.norm(z)
    P.close()


@pytest.mark.parametrize("dims", [(55, 127, 61), (63, 133, 70), (143, 301, 150)])
def test_coarse_diagonals_bit_exact_with_oracle(dims):
    """Level-1 diagonals (8,415, 11,305 and 111,111 nodes) on both sides of the 10,000 nodes from which a thread takes a node's three components."""
    import algorithmengineering_altproject_b200 as t3d
    from oracle.bindings import Oracle
    P = t3d.Problem(*dims)
    O = Oracle(*dims, red_mode=1, pow_mode=0, vol_mode=0, approx_mode=0)
    rng = np.random.default_rng(31)
    E = np.where(rng.random(P.ne) < 0.3, 1e-6, rng.uniform(0.05, 1.0, P.ne))
    P.make_diagonal_preconditioner_from_static(E)
    O.mg_build(E)
    for l in range(len(P.levels)):
        np.testing.assert_array_equal(P.mg_diag(l), O.mg_diag(l))
    P.close()
