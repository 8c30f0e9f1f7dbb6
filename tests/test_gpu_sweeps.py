"""Persistent triangular sweeps (forward and adjoint) against LAPACK on the oracle's operator.

Sizes: below, at and beside multiples of the 64-row blocks, more block rows than a chunk has
CTAs; columns: one, a partial and a full chunk of 4, one past a refinement group of 8, many
chunks, one past the 128 columns of a solve. Tolerance 1e-10 relative per column, the bar of the
other dense-solve tests (refined to an FP64 residual of 1e-12 or better on operators whose
condition numbers are below 1e2).
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def grid_cluster(count, lmax):
    g = np.stack(np.meshgrid(*[np.arange(5)] * 3, indexing="ij"), -1).reshape(-1, 3)[:count] * 0.62
    rng = np.random.default_rng(count)
    return lmax, 1.4, rng.uniform(0.15, 0.25, count), np.full(count, 2.5 + 0.05j), g + rng.uniform(-0.05, 0.05, g.shape)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("count,lmax,columns", [(1, 1, 1), (4, 2, 4), (2, 4, 5), (3, 4, 9), (7, 3, 2), (9, 4, 129),
                                                (30, 3, 33), (125, 2, 3)])
def test_solve_and_adjoint_match_lapack(ctx, precision, count, lmax, columns):
    import treams_b200 as t
    geom = grid_cluster(count, lmax)
    A, tb = oracle.cluster_operator(*geom)
    n = A.shape[0]
    rng = np.random.default_rng(columns)
    B, G = (np.asfortranarray(rng.standard_normal((n, columns)) + 1j * rng.standard_normal((n, columns)))
            for _ in range(2))
    f = t.sphere_cluster_factor(*geom, precision, ctx=ctx)
    X, certs = f.solve(B)
    Y, adj = f.solve_adjoint(G)
    f.close()
    for got, want in ((X, np.linalg.solve(A, oracle.apply_t(lmax, tb, B))), (Y, np.linalg.solve(A.conj().T, G))):
        err = np.linalg.norm(got - want, axis=0) / np.linalg.norm(want, axis=0)
        assert err.max() <= 1e-10
    for c in certs + adj:
        assert c.residual_norm <= 1e-12 * c.rhs_norm
