"""LU panels on clusters: factor quality over the panel's shapes.

Rows below, at and beside the steps of the cluster sizes (64 rows per CTA, 16 CTAs), one and several
clusters, last panels of every residue kind (a full sub-block, a partial one, less than one), on
densely packed spheres of high contrast at lmax 6 whose unscaled entries reach 1e5, so that rows do
interchange. A factor is judged by what its refinement needs: an FP64 factor reaches 1e-12 in one
sweep, a mixed one within 5 (the bound of the other dense tests), and the solutions of both agree
within 1e-9 of each other in the backward sense (their difference times A against T b).
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def dense_cluster(count, lmax, eps=6.0):
    rng = np.random.default_rng(100 * count + lmax)
    side = int(np.ceil(count ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:count] * 0.46
    return lmax, 2.6, rng.uniform(0.17, 0.21, count), rng.uniform(2, eps, count) + 0.1j, g + rng.uniform(-0.01, 0.01, g.shape)


@pytest.mark.parametrize("count,lmax", [(1, 1), (1, 3), (2, 3), (2, 5), (3, 6), (7, 6), (11, 6), (18, 5), (33, 6),
                                        (41, 5), (64, 4), (66, 4), (90, 6)])
def test_factors_of_every_panel_shape(ctx, count, lmax):
    import treams_b200 as t
    geom = dense_cluster(count, lmax)
    n = count * 2 * lmax * (lmax + 2)
    rng = np.random.default_rng(n)
    B = np.asfortranarray(rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2)))
    X = {}
    for precision, sweeps in (("fp64", 1), ("mixed", 5)):
        before = ctx.fallbacks
        f = t.sphere_cluster_factor(*geom, precision, ctx=ctx)
        X[precision], certs = f.solve(B)
        f.close()
        assert ctx.fallbacks == before
        for c in certs:
            assert c.residual_norm <= 1e-12 * c.rhs_norm and c.iterations <= sweeps
    d = t.cluster_apply(*geom, X["mixed"] - X["fp64"], ctx=ctx)
    tb = oracle.apply_t(lmax, t.mie_blocks(lmax, geom[1], geom[2], geom[3], ctx=ctx), B)
    assert np.linalg.norm(d) <= 1e-9 * np.linalg.norm(tb)
