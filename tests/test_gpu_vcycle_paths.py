"""Paths of the Adapted V-cycle that ordinary grids and moduli do not take, against the oracle, bit for bit: the coarsest
factor failing (Jacobi fallback inside the one-block tail and in the separate kernel) and recovering, spans of 2 from
the finest level on (mg_nondyadic = 0), and a coarsest inverse of 693 unknowns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def moduli(rng, n):
    return np.where(rng.random(n) < 0.3, 1e-6, rng.uniform(0.05, 1.0, n))


# 135 unknowns: solved in the tail, alone or below two more levels; 336: in the separate kernel
@pytest.mark.parametrize("dims", [(5, 9, 4), (30, 60, 30), (48, 96, 48)])
def test_failed_coarsest_factor(dims):
    import algorithmengineering_altproject_b200 as t3d
    from oracle.bindings import Oracle
    P = t3d.Problem(*dims)
    O = Oracle(*dims, red_mode=1, pow_mode=0, vol_mode=0, approx_mode=0)
    rng = np.random.default_rng(37)
    E, Ke = moduli(rng, P.ne), P.ke()
    for sign, ok in ((-1.0, 0), (1.0, 1)):   # a negative definite stiffness has no Cholesky factor
        P.set_ke(sign * Ke)
        O.set_ke(sign * Ke)
        P.make_diagonal_preconditioner_from_static(E)
        O.mg_build(E)
        assert P.info().coarse_cholesky_ok == ok
        r = rng.standard_normal(P.nf)
        z = P.vcycle(r)
        assert np.all(np.isfinite(z))
        np.testing.assert_array_equal(z, O.vcycle(r))
    P.close()


@pytest.mark.parametrize("dims", [(17, 40, 23), (30, 60, 30), (45, 101, 37)])
def test_spans_of_two_only(dims):
    import algorithmengineering_altproject_b200 as t3d
    from oracle.bindings import Oracle
    P = t3d.Problem(*dims, mg_nondyadic=0, precision=t3d.T3D_MIXED)
    O = Oracle(*dims, red_mode=1, pow_mode=0, vol_mode=0, approx_mode=0, nondyadic=0)
    assert P.levels[1][3] == 2 and len(P.levels) == O.nlev
    rng = np.random.default_rng(43)
    E = moduli(rng, P.ne)
    P.make_diagonal_preconditioner_from_static(E)
    O.mg_build(E)
    r = rng.standard_normal(P.nf).astype(np.float32).astype(np.float64)
    z = P.vcycle(r)
    np.testing.assert_array_equal(z, O.vcycle(r))
    assert np.linalg.norm(P.vcycle32(r) - z) <= 1e-5 * np.linalg.norm(z)
    P.close()


def test_coarsest_inverse_of_693_unknowns():
    import algorithmengineering_altproject_b200 as t3d
    from oracle.bindings import Oracle
    P = t3d.Problem(8, 40, 24)
    O = Oracle(8, 40, 24, red_mode=1, pow_mode=0, vol_mode=0, approx_mode=0)
    assert P.coarse_n == 693
    rng = np.random.default_rng(47)
    E = moduli(rng, P.ne)
    P.make_diagonal_preconditioner_from_static(E)
    O.mg_build(E)
    r = rng.standard_normal(P.nf)
    np.testing.assert_array_equal(P.vcycle(r), O.vcycle(r))
    P.close()
