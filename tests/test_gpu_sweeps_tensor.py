"""Triangular sweeps of three and more columns against those of the same columns one at a time.

Three columns and more run on the tensor-core sweep kernel, one and two on the other, so both forms
meet on the same factors: orders of one block, of whole blocks, of whole blocks and two rows; fewer and
more block rows than a chunk has CTAs and than its rings are deep; partial last chunks of one to
four columns. Both end at the rounding level of the refinement, some 1e-15 of the residual times
condition numbers below 1e3: 1e-11 relative per column.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("count,lmax,columns", [(1, 3, 3), (4, 2, 3), (8, 4, 4), (11, 2, 5), (13, 5, 6), (33, 1, 7),
                                                (40, 4, 67), (20, 3, 128)])
def test_chunks_match_single_columns(ctx, precision, count, lmax, columns):
    import treams_b200 as t
    rng = np.random.default_rng(count)
    g = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3)[:count] * 0.62
    geom = lmax, 1.4, rng.uniform(0.15, 0.25, count), np.full(count, 2.5 + 0.05j), g + rng.uniform(-0.05, 0.05, g.shape)
    n = count * 2 * lmax * (lmax + 2)
    B = np.asfortranarray(rng.standard_normal((n, columns)) + 1j * rng.standard_normal((n, columns)))
    f = t.sphere_cluster_factor(*geom, precision, ctx=ctx)
    for solve in (f.solve, f.solve_adjoint):
        X = np.asarray(solve(B)[0])
        for c in {0, 1, columns // 2, columns - 2, columns - 1}:
            want = np.asarray(solve(np.asfortranarray(B[:, c:c + 1]))[0])[:, 0]
            assert np.linalg.norm(X[:, c] - want) <= 1e-11 * np.linalg.norm(want)
    f.close()
