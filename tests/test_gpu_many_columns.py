"""More columns than a grid has rows (65,535), and columns whose packed inputs have no room.

The operator against the per-pair term sums, cross sections against calls of few columns. Products of
2 (2 lmax + 1) terms and sums over a few hundred modes: 1e-12 of the largest entry of a column, as in the
tests of the operator's forms.
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


@pytest.mark.parametrize("lmax", [2, 6])
def test_operator_beyond_a_grid(ctx, lmax, monkeypatch):
    import treams_b200 as t
    w = workloads.learned_cluster(seed=11, count=2)
    x = columns(2 * 2 * lmax * (lmax + 2), COLUMNS, lmax)
    y = t.cluster_apply(lmax, w.k0, w.radii, w.eps, w.positions, x, ctx=ctx)
    pick = np.r_[0:9, 4090:4100, COLUMNS - 12:COLUMNS]
    monkeypatch.setenv("TCU_APPLY", "terms")
    want = t.cluster_apply(lmax, w.k0, w.radii, w.eps, w.positions, np.asfortranarray(x[:, pick]), ctx=ctx)
    assert np.all(np.abs(y[:, pick] - want) <= 1e-12 * np.abs(want).max(axis=0))


@pytest.mark.parametrize("lmax", [1, 6])
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


@pytest.mark.parametrize("left", [30, 50, 80])
def test_operator_without_room_for_its_inputs(left):
    """4000 columns of two spheres at lmax 6: 25 MB of columns, 113 MB packed."""
    import torch
    import treams_b200 as t
    w = workloads.learned_cluster(seed=13, count=2)
    x = columns(2 * 96, 4000, 3)
    few = np.asfortranarray(x[:, ::500])
    own = t.Context(0)
    want = t.cluster_apply(6, w.k0, w.radii, w.eps, w.positions, few, ctx=own)
    sca, _ = t.cross_sections(6, w.k0, w.positions, few, few, ctx=own)
    own.close()
    own = t.Context(0)
    t.cluster_apply(6, w.k0, w.radii, w.eps, w.positions, few, ctx=own)  # its plan, while there is room
    held = []
    try:
        for _ in range(3):
            take = (torch.cuda.mem_get_info(0)[0] - (left << 20)) // (2 << 20) * (2 << 20)
            if take > 0:
                held.append(torch.empty(take, dtype=torch.uint8, device="cuda:0"))
        y = t.cluster_apply(6, w.k0, w.radii, w.eps, w.positions, x, ctx=own)
        if left >= 80:  # cross sections hold three sets of columns and 16 MB of partial sums: 53 MB
            got, _ = t.cross_sections(6, w.k0, w.positions, x, x, ctx=own)
    finally:
        held.clear()
        torch.cuda.empty_cache()
        own.close()
    assert np.all(np.abs(y[:, ::500] - want) <= 1e-12 * np.abs(want).max(axis=0))
    if left >= 80:
        assert np.all(np.abs(got[::500] - sca) <= 1e-12 * np.abs(sca).max())
