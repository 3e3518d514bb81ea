"""Blocks whose largest one picks a tiny solver (up to 8, 16 and 32 rows), both
sides of every limit, in calls whose descriptors are a kernel parameter and in
larger ones; random, degenerate and diagonal blocks.

Tolerance: 10 n eps for the residual and the orthogonality of a backward stable
solver, as for the other tiny blocks; eigenvalues against LAPACK the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [9, 200])
@pytest.mark.parametrize("nmax", [1, 2, 3, 7, 8, 9, 15, 16, 17, 32])
def test_every_tiny_solver(nmax, count):
    import nrgb
    rng = np.random.default_rng(100 * nmax + count)
    mats = []
    for i in range(count):
        n = nmax if i == 0 else int(rng.integers(1, nmax + 1))
        a = rng.standard_normal((n, n))
        a = a + a.T
        if i % 4 == 1:
            a = np.ones((n, n))
        elif i % 4 == 2:
            a = np.diag(np.diag(a))
        mats.append(a)
    ctx = nrgb.Context(0)
    try:
        ws, zs = ctx.syev_batched(mats)
    finally:
        ctx.close()
    for a, w, z in zip(mats, ws, zs):
        n = len(w)
        scale = max(1.0, np.max(np.abs(a)) * n)
        tol = 10 * n * 2.0 ** -52
        assert np.max(np.abs(w - np.linalg.eigvalsh(a))) <= tol * scale
        assert np.max(np.abs(z.T @ z - np.eye(n))) <= tol
        assert np.max(np.abs(a @ z - z * w[None, :])) <= tol * scale
