"""The Adapted V-cycle in its two forms -- separate kernels per level, and the one-block tail over the small levels --
against the oracle, bit for bit: grids whose hierarchy ends in a dense system the tail takes (135 unknowns), one it
does not (336 and, at 128x128x32, 729), and a Jacobi coarsest level; ragged sides and levels that divide no block."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(5, 9, 4), (17, 40, 23), (33, 67, 21), (30, 60, 30), (45, 101, 37), (48, 96, 48),
                                  (128, 128, 32)])
def test_adapted_vcycle_bit_exact_with_oracle(dims):
    import algorithmengineering_altproject_b200 as t3d
    from oracle.bindings import Oracle
    P = t3d.Problem(*dims)
    O = Oracle(*dims, red_mode=1, pow_mode=0, vol_mode=0, approx_mode=0)
    rng = np.random.default_rng(17)
    E = np.where(rng.random(P.ne) < 0.3, 1e-6, rng.uniform(0.05, 1.0, P.ne))
    P.make_diagonal_preconditioner_from_static(E)
    O.mg_build(E)
    for _ in range(2):
        r = rng.standard_normal(P.nf)
        np.testing.assert_array_equal(P.vcycle(r), O.vcycle(r))
    P.close()
