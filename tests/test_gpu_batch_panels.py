"""Panels of the batch's workers, which take 192 rows a CTA where a single factorization takes 64 to 128.

The sizes take half of the CTAs (1200 rows FP64, 1440 FP32: 8 instead of 16) or two clusters instead of three (5376
FP32). How the rows are dealt out changes neither a pivot nor an operation on a row, so a batch returns the very bits
of separate solves.
"""
import numpy as np
import pytest

import treams_b200 as t

pytestmark = pytest.mark.gpu


def cluster(count, lmax):
    rng = np.random.default_rng(count)
    side = int(np.ceil(count ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:count] * 0.55
    n = count * 2 * lmax * (lmax + 2)
    B = rng.standard_normal((n, 1)) + 1j * rng.standard_normal((n, 1))
    return lmax, 1.7, rng.uniform(0.15, 0.22, count), rng.uniform(2, 5, count) + 0.05j, g + rng.uniform(-0.02, 0.02, g.shape), B


@pytest.mark.parametrize("precision,sizes", [("fp64", [(40, 3), (18, 5)]), ("mixed", [(30, 4), (56, 6)])])
def test_batches_equal_separate_solves(ctx, precision, sizes):
    batch = [cluster(count, lmax) for count, lmax in sizes]
    X, _, _ = t.batch_solve(batch, precision, ctx=ctx)
    for Xi, (*geom, B) in zip(X, batch):
        f = t.sphere_cluster_factor(*geom, precision, ctx=ctx)
        assert np.array_equal(Xi, f.solve(B)[0])
        f.close()
