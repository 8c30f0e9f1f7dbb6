"""The lattice sums' order and reduction kernels over their shapes against the binary128 oracle.

Degrees from none to the largest (one pair to every warp of a group, one and both parities of
l - |m|), numbers of Bloch vectors beside the 32 of a warp and the 2, 4 and 8 of a CTA, in the plane
and off it, real and complex k, Bloch vectors of propagating and evanescent orders only. Bound as
in test_gpu_lattice.py: 1e-11 max(|D|, 1). A batch beyond one pass (64 MB of orders) equals its
parts bit for bit, since every sum has a fixed order.
"""
import numpy as np
import pytest

import oracle
from treams_b200 import lattice as tl

pytestmark = pytest.mark.gpu

LAT = np.array([[0.9, 0.1], [-0.2, 0.8]])


@pytest.mark.parametrize("lsum,nk", [(0, 1), (1, 31), (2, 33), (7, 5), (10, 66), (13, 3), (14, 9)])
@pytest.mark.parametrize("k,shift", [(3.3, None), (3.3, (0.2, -0.1, 0.0)), (2.9, (0.1, 0.3, 0.25)),
                                     (3.1 + 0.2j, (0.1, 0.0, 0.0)), (3.1 + 0.3j, (0.3, 0.1, -0.2))])
def test_tables_match_the_oracle(ctx, lsum, nk, k, shift):
    kps = np.random.default_rng(100 * lsum + nk).uniform(-3.5, 3.5, (nk, 2))
    D = tl.lsumsw2d_batch(lsum, k, LAT, kps, shift=shift, ctx=ctx)
    for i in sorted({0, nk // 2, nk - 1}):
        ref = oracle.lsumsw2d_table(lsum, k, LAT, kps[i], shift or (0.0, 0.0, 0.0))
        assert np.max(np.abs(D[i] - ref)) <= 1e-11 * max(1.0, np.max(np.abs(ref)))


def test_batches_beyond_one_pass_equal_their_parts(ctx):
    kps = np.random.default_rng(3).uniform(-3.5, 3.5, (6000, 2))
    whole = tl.lsumsw2d_batch(14, 2.9, LAT, kps, shift=(0.1, 0.3, 0.25), ctx=ctx)
    parts = np.concatenate([tl.lsumsw2d_batch(14, 2.9, LAT, kps[i:i + 1000], shift=(0.1, 0.3, 0.25), ctx=ctx)
                            for i in range(0, 6000, 1000)])
    # the reciprocal cutoff follows the largest Bloch vector of a call: orders beyond 1e-20 only
    assert np.max(np.abs(whole - parts)) <= 1e-15 * np.max(np.abs(parts))
