"""Every bounded device wait gives up on what never comes: grid barrier, cluster panel's message and word,
sweeps' entry and ring, trailing update's ring, stored product's ring.

The self-test runs them one after the other, each with the given limit, and names one that did not give
up; seven waits of 50 ms take 0.35 s, and each ends within a few polls of its limit.
"""
import time

import pytest

pytestmark = pytest.mark.gpu

WAITS, LIMIT = 7, 0.05


def test_every_wait_gives_up_at_its_limit(ctx):
    import treams_b200 as t
    with pytest.raises(t.TreamsCudaError, match="a device-side wait gave up"):
        ctx.wait_selftest(0.0)
    t0 = time.perf_counter()
    with pytest.raises(t.TreamsCudaError, match="a device-side wait gave up"):
        ctx.wait_selftest(LIMIT)
    elapsed = time.perf_counter() - t0
    assert WAITS * LIMIT <= elapsed <= WAITS * LIMIT + 0.5
