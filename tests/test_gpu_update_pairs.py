"""Trailing updates by CTA pairs: tiles whose second CTA has few rows or none.

Orders that leave 4, 64, 66, 128, 130 and 384 complex rows right of the first panel (a pair takes 128 of
them, each CTA 64), and a few past the second one, so that the second CTA of the last pair lies beside,
on and inside the matrix edge, and the second half of the columns too. Bound as for the update's other
tests: 4 * 2^-17 of |T b| unrefined.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,lmax", [(22, 1), (12, 2), (32, 1), (97, 1), (43, 1), (16, 2), (64, 2), (66, 2), (37, 3)])
def test_unrefined_residual(ctx, count, lmax):
    import treams_b200 as t
    rng = np.random.default_rng(count)
    side = int(np.ceil(count ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:count] * 0.6
    geom = (lmax, 2.0, rng.uniform(0.15, 0.2, count), rng.uniform(2, 3, count) + 0.05j,
            g + rng.uniform(-0.01, 0.01, g.shape))
    n = count * 2 * lmax * (lmax + 2)
    b = np.asfortranarray(rng.standard_normal((n, 1)) + 1j * rng.standard_normal((n, 1)))
    f = t.sphere_cluster_factor(*geom, "mixed", ctx=ctx)
    try:
        ctx.set_refinement(1e300, 1e300)
        c = f.solve(b)[1][0]
        assert c.residual_norm <= 4 * 2.0**-17 * c.rhs_norm
    finally:
        ctx.set_refinement(1e-13, 1e-12)
        f.close()
