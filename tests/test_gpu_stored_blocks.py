"""The stored product leaves out blocks of its table that no term reads: every entry of the operator.

Unit vectors as inputs, so that each (destination mode, source mode) pair is one output, against the
per-pair term sums; counts that leave a destination block partly filled and one chunk of sources.
An entry is a sum of at most 2 (2 lmax + 1) products, the same ones in both forms: rounding stays
below 30 * 2^-53 of the largest term, and a column's largest entry is at least a tenth of the largest
term of its well-separated pairs, so 1e-13 of it is a bound with room; an entry left out is missing
altogether.
"""
import numpy as np
import pytest

from treams_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax,count", [(2, 6), (3, 3), (4, 2), (5, 2), (6, 2), (7, 2), (3, 17)])
def test_every_entry(ctx, lmax, count, monkeypatch):
    import treams_b200 as t
    w = workloads.learned_cluster(seed=40 + lmax, count=count)
    n = count * 2 * lmax * (lmax + 2)
    x = np.asfortranarray(np.eye(n, dtype=complex))
    got = {}
    for form in ("stored", "terms"):
        monkeypatch.setenv("TCU_APPLY", form)
        got[form] = t.cluster_apply(lmax, w.k0, w.radii, w.eps, w.positions, x, ctx=ctx) - x
    scale = np.abs(got["terms"]).max(axis=0)
    assert np.all(np.abs(got["stored"] - got["terms"]) <= 1e-13 * scale)
