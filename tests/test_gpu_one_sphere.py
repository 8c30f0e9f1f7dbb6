"""A cluster of one sphere couples to nothing: no tables of pairs are built for it, at any degree (up to 16 columns;
beyond, the product over empty tables is the faster one)."""
import numpy as np
import pytest

import treams_b200 as t

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax", [1, 2, 5, 6, 7])
@pytest.mark.parametrize("columns", [1, 3, 16])
def test_one_sphere_launches_what_the_plain_form_does(ctx, lmax, columns, monkeypatch):
    geom = (lmax, 1.5, [0.3], [3 + 0.05j], np.zeros((1, 3)))
    n = 2 * lmax * (lmax + 2)
    rng = np.random.default_rng(lmax)
    x = rng.standard_normal((n, columns)) + 1j * rng.standard_normal((n, columns))
    counts, values = [], []
    for form in ("fly", None):
        if form:
            monkeypatch.setenv("TCU_APPLY", form)
        else:
            monkeypatch.delenv("TCU_APPLY")
        calls = [lambda: t.cluster_apply(*geom, x, ctx=ctx), lambda: np.array(t.cross_sections(lmax, 1.5, geom[4], x, x, ctx=ctx)),
                 lambda: t.SphereCluster(*geom, ctx=ctx).solve(x).value]
        for call in calls:
            before = ctx.launches
            values.append(call())
            counts.append(ctx.launches - before)
    assert counts[:3] == counts[3:]
    for a, b in zip(values[:3], values[3:]):
        assert np.array_equal(a, b)
    assert np.array_equal(values[0], x)
