"""Cross sections of many columns at once: their sums have scratch for every column.

Against the oracle column by column; 1e-12 of the sum's natural scale, one application of the FP64
operator and a dot product, as for few columns.
"""
import numpy as np
import pytest

import oracle
from treams_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax,count,columns", [(3, 9, 5), (2, 7, 33), (6, 3, 9), (4, 1, 70)])
def test_every_column(ctx, lmax, count, columns):
    import treams_b200 as t
    w = workloads.learned_cluster(seed=9 + lmax, count=count)
    n = count * 2 * lmax * (lmax + 2)
    rng = np.random.default_rng(columns)
    x, b = (rng.standard_normal((n, columns)) + 1j * rng.standard_normal((n, columns)) for _ in range(2))
    sca, ext = t.cross_sections(lmax, w.k0, w.positions, x, b, ctx=ctx)
    for c in {0, 1, columns // 2, columns - 1}:
        so, eo = oracle.cross_sections(lmax, w.k0, w.positions, x[:, c], b[:, c])
        scale = np.linalg.norm(x[:, c]) ** 2 / w.k0**2
        assert abs(sca[c] - so) <= 1e-12 * max(abs(so), scale) and abs(ext[c] - eo) <= 1e-12 * max(abs(eo), scale)
