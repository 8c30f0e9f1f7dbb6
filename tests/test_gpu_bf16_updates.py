"""Trailing updates of the mixed LU in three bfloat16 passes: factor quality without refinement.

Orders with every kind of remainder of the update: less than one panel right of the first, one and
two panels per update, last panels and last 32-element K chunks partly filled, row tiles of 64 and
column tiles of 256 partly filled. Each term of an update carries a relative error of about 2^-17
(lo * lo dropped, lo rounded), and the operators are close to the unit matrix after equilibration,
so |L||U| is of the order of |A| and the unrefined residual stays below 4 * 2^-17 of |T b|.
Refined to 1e-13, the solution ends at the FP64 rounding level, well below 1e-14.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def grid_cluster(count, lmax):
    rng = np.random.default_rng(1000 * count + lmax)
    side = int(np.ceil(count ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:count] * 0.6
    return lmax, 2.0, rng.uniform(0.15, 0.2, count), rng.uniform(2, 3, count) + 0.05j, g + rng.uniform(-0.01, 0.01, g.shape)


@pytest.mark.parametrize("count,lmax", [(9, 3), (8, 4), (5, 5), (4, 6), (16, 4), (43, 3), (17, 6), (55, 5), (100, 4)])
def test_unrefined_and_refined_residuals(ctx, count, lmax):
    import treams_b200 as t
    geom = grid_cluster(count, lmax)
    n = count * 2 * lmax * (lmax + 2)
    rng = np.random.default_rng(n)
    B = np.asfortranarray(rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2)))
    f = t.sphere_cluster_factor(*geom, "mixed", ctx=ctx)
    try:
        for target, bound in ((1e300, 4 * 2.0**-17), (1e-13, 1e-14)):
            ctx.set_refinement(target, 1e300)
            for c in f.solve(B)[1]:
                assert c.residual_norm <= bound * c.rhs_norm
    finally:
        ctx.set_refinement(1e-13, 1e-12)
        f.close()
