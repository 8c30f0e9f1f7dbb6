"""A timeout is reported once: a factor whose earlier solve gave up solves again.

The self-test leaves the sweeps' give-up in the status word of every live factor, as a solve whose wait
ran out would. 1e-10 relative against LAPACK on the oracle's operator, the bar of the other dense tests.
"""
import numpy as np
import pytest

import oracle
from treams_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("columns", [1, 5])
def test_factor_solves_after_a_timeout(ctx, precision, columns):
    import treams_b200 as t
    w = workloads.small_cluster()
    geom = (w.lmax, w.k0, w.radii, w.eps, w.positions)
    A, tb = oracle.cluster_operator(*geom)
    rng = np.random.default_rng(columns)
    B = np.asfortranarray(rng.standard_normal((A.shape[0], columns)) + 1j * rng.standard_normal((A.shape[0], columns)))
    f = t.sphere_cluster_factor(*geom, precision, ctx=ctx)
    try:
        with pytest.raises(t.TreamsCudaError, match="gave up"):
            ctx.wait_selftest(0.01)
        X, _ = f.solve(B)
        Y, _ = f.solve_adjoint(B)
    finally:
        f.close()
    for got, want in ((X, np.linalg.solve(A, oracle.apply_t(w.lmax, tb, B))), (Y, np.linalg.solve(A.conj().T, B))):
        assert np.all(np.linalg.norm(got - want, axis=0) <= 1e-10 * np.linalg.norm(want, axis=0))
