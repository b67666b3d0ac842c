"""The OC bisection's volume sums against the oracle, bit for bit, in both summation orders: element counts around
the edges of the parallel evaluation of the reference's float order (fewer than one block of 8, one group of 8192
elements, one more, remainders of 1..7) and densities that make the chains round awkwardly (exact halfway cases,
all equal, all at the bounds)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(1, 2, 3), (2, 4, 1), (3, 5, 7), (16, 32, 16), (25, 41, 8), (20, 41, 10), (48, 96, 33)]


def fields(kind, n, rng):
    if kind == "random":
        x = rng.uniform(1e-3, 1.0, n)
        dc = -np.exp(2.0 * rng.standard_normal(n))
    elif kind == "halfway":   # candidates clamp to x +- 0.2 or stay at dyadic values: ties in the float sums
        x = rng.integers(1, 257, n) / 256.0
        dc = -np.where(rng.uniform(size=n) < 0.5, 1.0, 0.25)
    elif kind == "equal":
        x, dc = np.full(n, 0.12), np.full(n, -1.0)
    else:                     # near-binary design
        x = np.where(rng.uniform(size=n) < 0.12, 1.0, 1e-3)
        dc = -x * rng.uniform(0.5, 2.0, n)
    return x.astype(np.float32), dc.astype(np.float32)


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("dims", DIMS)
def test_oc_update_bit_exact_with_oracle(dims, order):
    import algorithmengineering_altproject_b200 as t3d
    from oracle.bindings import Oracle
    P = t3d.Problem(*dims, oc_sum_order=order)
    O = Oracle(*dims, red_mode=1, pow_mode=0, vol_mode=2 if order else 0, approx_mode=0)
    rng = np.random.default_rng(11)
    for kind in ("random", "halfway", "equal", "binary"):
        x, dc = fields(kind, P.ne, rng)
        for V0 in (0.08, 0.3):
            xg, chg, lmg, nbg = P.oc_update(x, dc, V0)
            xo, cho, lmo, nbo = O.oc(x, dc, V0)
            assert (nbg, lmg, chg) == (nbo, lmo, cho), (kind, V0)
            np.testing.assert_array_equal(xg.view(np.uint32), xo.view(np.uint32))
    P.close()
