"""Dense solves where device memory is nearly used up.

Stored pair tables and many columns side by side are there for speed: wherever a factor without tables and
eight columns at a time have room, the default forms and 128 columns have to succeed too, with the same
solution (1e-10 relative, the bar of the other dense tests). Memory is taken away in steps of 2 MB, the
allocator's granularity, around the bytes that the factor and its solve need; every size runs with a
context of its own, so that no pool keeps anything. The default forms get two steps more than the plain
ones: tables that gave way leave a hole inside an allocator's block, which a larger buffer cannot use.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

MB = 1 << 20


def cluster(lmax, count):
    g = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3)[:count] * 0.62
    rng = np.random.default_rng(count)
    return lmax, 1.4, rng.uniform(0.15, 0.25, count), np.full(count, 2.5 + 0.05j), g + rng.uniform(-0.05, 0.05, g.shape)


def attempt(t, geom, precision, B):
    """The solutions, or None without room."""
    own = t.Context(0)
    try:
        f = t.sphere_cluster_factor(*geom, precision, ctx=own)
        X, _ = f.solve(B)
        Y, _ = f.solve_adjoint(B)
        return X, Y
    except MemoryError:
        return None
    finally:
        own.close()


@pytest.mark.parametrize("precision,lmax,count", [("mixed", 6, 12), ("fp64", 4, 30)])
def test_speed_forms_fit_where_the_plain_ones_do(precision, lmax, count, monkeypatch):
    import torch
    import treams_b200 as t
    geom = cluster(lmax, count)
    A, tb = oracle.cluster_operator(*geom)
    n = A.shape[0]
    rng = np.random.default_rng(n)
    B = np.asfortranarray(rng.standard_normal((n, 128)) + 1j * rng.standard_normal((n, 128)))
    want = np.linalg.solve(A, oracle.apply_t(lmax, tb, B)), np.linalg.solve(A.conj().T, B)

    def check(got):
        for g, w in zip(got, want):
            assert np.all(np.linalg.norm(g - w, axis=0) <= 1e-10 * np.linalg.norm(w, axis=0))

    for form in ("fly", "stored"):  # every kernel is loaded while there is room
        monkeypatch.setenv("TCU_APPLY", form)
        check(attempt(t, geom, precision, B))
    matrix = n * n * (16 if precision == "fp64" else 8)
    fitted = refused = 0
    plain_fits = []
    for extra in range(0, 120, 2):
        torch.cuda.empty_cache()
        held = []
        try:
            for _ in range(3):  # the first block leaves a little more than asked for
                free = torch.cuda.mem_get_info(0)[0]
                take = (free - matrix - extra * MB) // (2 * MB) * (2 * MB)
                if take > 0:
                    held.append(torch.empty(take, dtype=torch.uint8, device="cuda:0"))
            monkeypatch.setenv("TCU_APPLY", "fly")
            plain_fits.append(attempt(t, geom, precision, np.asfortranarray(B[:, :8])) is not None)
            monkeypatch.delenv("TCU_APPLY")
            got = attempt(t, geom, precision, B)
        finally:
            held.clear()
            torch.cuda.empty_cache()
        if got is not None:
            check(got)
        if len(plain_fits) < 3 or not plain_fits[-3]:
            refused += not plain_fits[-1]
            continue
        assert got is not None, f"{extra} MB beside the matrix: the plain forms fit in {extra - 4}, the default ones not"
        fitted += 1
        if fitted == 6:
            break
    assert fitted and refused
