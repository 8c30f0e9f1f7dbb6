"""Columns of one solve that converge at different sweeps, against LAPACK on the oracle's operator.

Zero columns are done after the first sweep, the others take more, so groups of 8 leave the packed columns at
the front, in the middle and at the end, with a narrow last group in either state; three residuals fall back
at once. 1e-10 relative per column, the bar of the other dense tests; zero columns give exact zeros.
"""
import numpy as np
import pytest

import oracle
from treams_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("columns,zero_groups", [(20, [0]), (20, [1]), (20, [2]), (33, [0, 2]), (33, [1, 4]),
                                                 (128, list(range(1, 16))), (129, [0, 15]), (16, [0, 1])])
def test_groups_leave_at_different_sweeps(ctx, precision, columns, zero_groups):
    import treams_b200 as t
    w = workloads.small_cluster()
    geom = (w.lmax, w.k0, w.radii, w.eps, w.positions)
    A, tb = oracle.cluster_operator(*geom)
    n = A.shape[0]
    rng = np.random.default_rng(columns)
    B = np.asfortranarray(rng.standard_normal((n, columns)) + 1j * rng.standard_normal((n, columns)))
    zero = np.isin(np.arange(columns) // 8, zero_groups)
    B[:, zero] = 0.0
    f = t.sphere_cluster_factor(*geom, precision, ctx=ctx)
    try:
        X, certs = f.solve(B)
        Y, adj = f.solve_adjoint(B)
        G, pull = f.pullback_incident(B)
    finally:
        f.close()
    Yo = np.linalg.solve(A.conj().T, B)
    T = oracle.apply_t(w.lmax, tb, np.eye(n, dtype=complex))
    for got, want, cert in ((X, np.linalg.solve(A, oracle.apply_t(w.lmax, tb, B)), certs), (Y, Yo, adj),
                            (G, T.conj().T @ Yo, pull)):
        assert not got[:, zero].any()
        norm = np.linalg.norm(want[:, ~zero], axis=0)
        assert np.all(np.linalg.norm(got[:, ~zero] - want[:, ~zero], axis=0) <= 1e-10 * norm)
        for c, z in zip(cert, zero):
            assert c.iterations == 1 if z else c.residual_norm <= 1e-12 * c.rhs_norm
        if precision == "mixed":
            assert all(c.iterations > 1 for c, z in zip(cert, zero) if not z)


def test_a_stalled_group_falls_back_beside_others(ctx):
    """Limits under which every nonzero group of a mixed factor stalls: the others' columns stay as they are."""
    import treams_b200 as t
    w = workloads.small_cluster()
    geom = (w.lmax, w.k0, w.radii, w.eps, w.positions)
    A, tb = oracle.cluster_operator(*geom)
    rng = np.random.default_rng(5)
    B = np.asfortranarray(rng.standard_normal((A.shape[0], 19)) + 1j * rng.standard_normal((A.shape[0], 19)))
    B[:, 8:16] = 0.0
    own = t.Context(0)
    own.set_refinement(1e-18, 1e-18)
    f = t.sphere_cluster_factor(*geom, "mixed", ctx=own)
    try:
        X, certs = f.solve(B)
        Y, _ = f.solve_adjoint(B)
    finally:
        f.close()
        own.close()
    for got, want in ((X, np.linalg.solve(A, oracle.apply_t(w.lmax, tb, B))), (Y, np.linalg.solve(A.conj().T, B))):
        assert not got[:, 8:16].any()
        for c in list(range(8)) + [16, 17, 18]:
            assert np.linalg.norm(got[:, c] - want[:, c]) <= 1e-10 * np.linalg.norm(want[:, c])
