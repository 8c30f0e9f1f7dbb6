"""The stored product at lmax 6 and 7: last tiles cut into pieces of the source chunks.

Counts and columns whose tiles (two or four per destination and column) end in a last wave of 2, 4, 40
or 74 of 148 SMs, within one column and across the last ones, with as many pieces as chunks, fewer
chunks than pieces, and one chunk (no pieces), against the per-pair term sums. The bound is that of
the other forms of the operator, 1e-13 relative for FP64 sums of a few thousand terms.
"""
import numpy as np
import pytest

from treams_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax,count,columns", [(6, 75, 1), (6, 20, 1), (6, 37, 3), (6, 50, 3), (6, 9, 1), (7, 38, 1),
                                                (7, 10, 1), (7, 39, 2)])
def test_tail_pieces(ctx, lmax, count, columns, monkeypatch):
    import treams_b200 as t
    w = workloads.learned_cluster(seed=70 + lmax + count, count=count)
    n = count * 2 * lmax * (lmax + 2)
    rng = np.random.default_rng(n)
    x = np.asfortranarray(rng.standard_normal((n, columns)) + 1j * rng.standard_normal((n, columns)))
    got = {}
    for form in ("stored", "terms"):
        monkeypatch.setenv("TCU_APPLY", form)
        got[form] = t.cluster_apply(lmax, w.k0, w.radii, w.eps, w.positions, x, ctx=ctx)
    for c in range(columns):
        assert np.linalg.norm(got["stored"][:, c] - got["terms"][:, c]) <= 1e-13 * np.linalg.norm(got["terms"][:, c])
