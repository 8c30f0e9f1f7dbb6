"""Large results through the context's pinned ring equal the plain copies.

Sizes around the 32 MB where the ring takes over and around its 2 MB slots (the result of nk Bloch
vectors at lmax 3 is nk * 14,400 bytes), into fresh and into reused host memory; each call against
the same Bloch vectors solved in small calls, which copy plainly. The kernels are deterministic, so
the values are equal bit for bit (one cutoff radius: the largest Bloch vector is in every call).
"""
import numpy as np
import pytest

from treams_b200 import lattice as tl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk", [2330, 2331, 2477, 5000])
def test_array_results_equal_small_calls(ctx, nk):
    lat = np.array([[0.74, 0.0], [0.02, 0.74]])
    kps = np.random.default_rng(nk).uniform(-4.0, 4.0, (nk, 2))
    kps[::500] = (4.0, 4.0)
    big = tl.array_solve_batch(3, 4.0, 0.2, 6.0 + 0.1j, lat, kps, ctx=ctx)
    for i in range(0, nk, 500):
        part = tl.array_solve_batch(3, 4.0, 0.2, 6.0 + 0.1j, lat, kps[i:i + 500], ctx=ctx)
        assert np.array_equal(big[i:i + 500], part)
