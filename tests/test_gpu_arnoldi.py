"""Arnoldi steps with one wait for the host: long bases and every group of their columns.

A resonant cluster that needs some hundred steps, with restart lengths below, at and above the 64
columns of one group of the Gram-Schmidt kernel and of two. The residual is taken again from the
operator itself: rtol plus its own rounding (some thousand FP64 terms, far below 1e-12 of the
right-hand side).
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("restart", [5, 64, 65, 130, 400])
def test_residual_for_every_basis_length(ctx, restart):
    import treams_b200 as t
    rng = np.random.default_rng(125)
    g = np.stack(np.meshgrid(*[np.arange(5)] * 3, indexing="ij"), -1).reshape(-1, 3) * 0.46
    geom = 3, 3.6, rng.uniform(0.2, 0.21, 125), np.full(125, 12.0 + 0.001j), g + rng.uniform(-0.005, 0.005, g.shape)
    n = 125 * 30
    b = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    rtol = 1e-6 if restart < 64 else 1e-10
    s = t.SphereCluster(*geom, ctx=ctx).solve(b, rtol=rtol, restart=restart, max_iterations=3000)
    tb = oracle.apply_t(3, t.mie_blocks(3, geom[1], geom[2], geom[3], ctx=ctx), b[:, None])[:, 0]
    x = np.asarray(s.value).reshape(n)
    r = tb - t.cluster_apply(*geom, x[:, None], ctx=ctx)[:, 0]
    assert s.convergence[0].residual_norm <= rtol * s.convergence[0].rhs_norm
    assert np.linalg.norm(r) <= (rtol + 1e-12) * np.linalg.norm(tb)
