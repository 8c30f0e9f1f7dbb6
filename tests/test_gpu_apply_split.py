"""The stored-table operator at lmax 6 and 7 (its product split over helicities and source halves).

Counts beside the 16-source chunks and the 32-source build chunks, one and several columns, the
outgoing operator and the regular operator of the cross sections against the oracle, and GMRES
against the term sums. Bounds as for lmax 2..5: 1e-13 relative for one application (FP64
sums of a few thousand terms), 1e-12 for the cross sections (one application and a dot product).
"""
import numpy as np
import pytest

import oracle
from treams_b200 import workloads

pytestmark = pytest.mark.gpu


def _cluster(lmax, count):
    return workloads.learned_cluster(seed=600 + 10 * lmax + count, count=count)


@pytest.mark.parametrize("lmax", [6, 7])
@pytest.mark.parametrize("count,columns", [(1, 1), (2, 3), (16, 1), (33, 2), (49, 9)])
def test_operator_matches_the_oracle(ctx, lmax, count, columns):
    import treams_b200 as t
    w = _cluster(lmax, count)
    n = count * 2 * lmax * (lmax + 2)
    rng = np.random.default_rng(count)
    x = rng.standard_normal((n, columns)) + 1j * rng.standard_normal((n, columns))
    got = t.cluster_apply(lmax, w.k0, w.radii, w.eps, w.positions, x, ctx=ctx)
    want = oracle.iterative_apply(lmax, w.k0, w.radii, w.eps, w.positions, x)
    assert np.linalg.norm(got - want) <= 1e-13 * np.linalg.norm(want)


@pytest.mark.parametrize("lmax", [6, 7])
def test_cross_sections_match_the_oracle(ctx, lmax):
    import treams_b200 as t
    w = _cluster(lmax, 18)
    n = 18 * 2 * lmax * (lmax + 2)
    rng = np.random.default_rng(lmax)
    x, b = (rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2)) for _ in range(2))
    sca, ext = t.cross_sections(lmax, w.k0, w.positions, x, b, ctx=ctx)
    for c in range(2):
        so, eo = oracle.cross_sections(lmax, w.k0, w.positions, x[:, c], b[:, c])
        scale = np.linalg.norm(x[:, c]) ** 2 / w.k0**2
        assert abs(sca[c] - so) <= 1e-12 * max(abs(so), scale) and abs(ext[c] - eo) <= 1e-12 * max(abs(eo), scale)


@pytest.mark.parametrize("lmax", [6, 7])
def test_gmres_matches_the_term_sums(ctx, lmax, monkeypatch):
    import treams_b200 as t
    w = _cluster(lmax, 40)
    c = t.SphereCluster(lmax, w.k0, w.radii, w.eps, w.positions, ctx=ctx)
    B = t.plane_wave_expansion(lmax, w.positions, w.kvecs, w.pols, ctx=ctx)
    monkeypatch.delenv("TCU_APPLY", raising=False)
    s1 = c.solve(B, rtol=1e-12, restart=40, max_iterations=400)
    monkeypatch.setenv("TCU_APPLY", "terms")
    s2 = c.solve(B, rtol=1e-12, restart=40, max_iterations=400)
    assert [v.iterations for v in s1.convergence] == [v.iterations for v in s2.convergence]
    assert np.linalg.norm(s1.value - s2.value) <= 1e-11 * np.linalg.norm(s2.value)
