"""Batches give back what their threads take: device memory after many calls of the same batch.

Every call starts new host threads, whose mixed factorizations use a stream of their own. 60 calls with 4 threads
that kept it would hold 150 MB; the pools are filled by the first calls, so a quarter of that is the bound.
"""
import numpy as np
import pytest
import torch

import treams_b200 as t

pytestmark = pytest.mark.gpu


def test_batches_do_not_accumulate_device_memory(ctx):
    rng = np.random.default_rng(11)
    batch = []
    for count in (6, 7, 8, 9, 10, 11):
        x = np.zeros((count, 3))
        x[:, 0] = 0.8 * np.arange(count)
        n = count * 30
        batch.append((3, 1.5, rng.uniform(0.2, 0.3, count), np.full(count, 3 + 0.05j), x,
                      rng.standard_normal((n, 1)) + 1j * rng.standard_normal((n, 1))))

    def used():
        free, total = torch.cuda.mem_get_info()
        return total - free

    for _ in range(4):
        t.batch_solve(batch, "mixed", ctx=ctx)
    before = used()
    for _ in range(60):
        t.batch_solve(batch, "mixed", ctx=ctx)
    assert used() - before <= 37 << 20
