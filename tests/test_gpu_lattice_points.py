"""Lattice sums over more real-space points than one CTA's shared memory would hold, against the binary128 oracle.

Small cells (k a about 0.4) at a small Ewald split: 10,400 to 12,300 points within the cutoff, beyond the 8,320
to 11,392 that a kernel with a phase per point in shared memory could take. The oracle sums at its own split.
Per degree 1e-10 of the degree's largest entry: 12,000 terms of at most e^2 times the sum (1/(2 eta^2) = 2)
round to some 1e-13 of it; over all degrees the 1e-11 max(|D|, 1) of the other lattice tests.
"""
import numpy as np
import pytest

import oracle
from treams_b200 import lattice as tl

pytestmark = pytest.mark.gpu

KPARS = np.array([[0.3, 0.1], [-1.7, 2.3], [0.9, -0.4]])


@pytest.mark.parametrize("lsum,a,k,shift", [
    (4, 0.36, 1.0, None), (12, 0.43, 1.0, None), (8, 0.40, 1.0, (0.10, 0.05, 0.08)), (14, 0.45, 1.0, (0.05, 0.10, 0.10)),
    (14, 0.45, 1.0, None), (8, 0.42, 1.0 + 0.05j, None), (12, 0.45, 1.0 + 0.05j, (0.10, 0.05, 0.08))])
def test_many_points_match_the_oracle(ctx, lsum, a, k, shift):
    lat = np.array([[a, 0.0], [0.0, a]])
    D = tl.lsumsw2d_batch(lsum, k, lat, KPARS, eta=0.5, shift=shift, ctx=ctx)
    for got, kp in zip(D, KPARS):
        ref = oracle.lsumsw2d_table(lsum, k, lat, kp, shift or (0.0, 0.0, 0.0))
        assert np.max(np.abs(got - ref)) <= 1e-11 * max(1.0, np.max(np.abs(ref)))
        for l in range(lsum + 1):
            s = slice(l * l, (l + 1) ** 2)
            assert np.max(np.abs(got[s] - ref[s])) <= 1e-10 * np.max(np.abs(ref[s]))


def test_a_lattice_beyond_129_points_a_side_is_refused(ctx):
    with pytest.raises(ValueError, match="elongated"):
        tl.lsumsw2d_batch(4, 1.0, np.array([[0.2, 0.0], [0.0, 0.2]]), KPARS, eta=0.5, ctx=ctx)
