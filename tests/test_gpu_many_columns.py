"""More columns than a grid has rows (65,535).

Cross sections against calls of few columns: sums over a few hundred modes, 1e-12 of their terms' bound.
"""
import numpy as np
import pytest

from treams_b200 import workloads

pytestmark = pytest.mark.gpu

COLUMNS = 65540


def columns(n, p, seed):
    rng = np.random.default_rng(seed)
    x = np.empty((n, p), complex, order="F")
    x.real, x.imag = rng.standard_normal((p, n)).T, rng.standard_normal((p, n)).T
    return x


@pytest.mark.parametrize("lmax", [1])
def test_cross_sections_beyond_a_grid(ctx, lmax):
    import treams_b200 as t
    w = workloads.learned_cluster(seed=12, count=2)
    n = 2 * 2 * lmax * (lmax + 2)
    x, b = columns(n, COLUMNS, 1), columns(n, COLUMNS, 2)
    sca, ext = t.cross_sections(lmax, w.k0, w.positions, x, b, ctx=ctx)
    pick = np.r_[0:5, COLUMNS - 5:COLUMNS]
    ps, pe = t.cross_sections(lmax, w.k0, w.positions, np.asfortranarray(x[:, pick]), np.asfortranarray(b[:, pick]),
                              ctx=ctx)
    scale = np.abs(x[:, pick]).max(axis=0) ** 2 * n / w.k0 ** 2
    assert np.all(np.abs(sca[pick] - ps) <= 1e-12 * scale) and np.all(np.abs(ext[pick] - pe) <= 1e-12 * scale)
