"""Divide and conquer inside one CTA: blocks solved whole (n <= 32), subtrees
of every depth and size around its limits (64, 128 rows), spectra that deflate
in each way (tight clusters, multiple eigenvalues, decoupled rows, a constant
diagonal), against LAPACK; a block with an entry that is not a number is an error."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = list(range(1, 40)) + [47, 48, 63, 64, 65, 66, 95, 96, 127, 128, 129, 130, 191, 255, 256, 257, 300, 513]


def _block(kind, n, rng):
    if kind == "gaussian":
        a = rng.standard_normal((n, n))
        return a + a.T
    if kind == "tridiagonal":  # constant diagonal and couplings: every tearing sees equal halves
        return 2.0 * np.eye(n) + np.diag(np.ones(n - 1), 1) + np.diag(np.ones(n - 1), -1)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    if kind == "multiple":
        w = rng.integers(0, max(2, n // 6), n).astype(float)
    elif kind == "clusters":
        w = rng.integers(0, max(2, n // 5), n) + 1e-13 * rng.standard_normal(n)
    elif kind == "logspaced":
        w = np.logspace(-12, 1, n) * rng.choice([-1.0, 1.0], n)
    else:  # decoupled
        a = rng.standard_normal((n, n))
        a = a + a.T
        cut = rng.random((n, n)) < 0.7
        a[cut | cut.T] = 0.0
        return a
    a = (q * w) @ q.T
    return (a + a.T) / 2


@pytest.mark.parametrize("kind", ["gaussian", "tridiagonal", "multiple", "clusters", "logspaced", "decoupled"])
def test_subtrees_against_lapack(kind):
    import nrgb
    rng = np.random.default_rng(len(kind))
    mats = [_block(kind, n, rng) for n in SIZES]
    ctx = nrgb.Context(0)
    try:
        ws, zs = ctx.syev_batched(mats)
    finally:
        ctx.close()
    for a, w, z in zip(mats, ws, zs):
        n = a.shape[0]
        ref = np.linalg.eigvalsh(a)
        tol = 1e-13 * max(n, 10) * max(np.max(np.abs(ref)), 1e-300)
        assert np.max(np.abs(w - ref)) <= tol, ("eigenvalues", kind, n)
        assert np.max(np.abs(a @ z - z * w)) <= tol, ("residual", kind, n)
        assert np.max(np.abs(z.T @ z - np.eye(n))) <= 1e-13 * max(n, 10), ("orthogonality", kind, n)


@pytest.mark.parametrize("n", [2, 5, 20, 33, 64, 100, 128])
def test_not_a_number_is_an_error(n):
    import nrgb
    a = np.random.default_rng(n).standard_normal((n, n))
    a = a + a.T
    a[n // 2, n // 2 - 1] = a[n // 2 - 1, n // 2] = np.nan
    ctx = nrgb.Context(0)
    try:
        with pytest.raises(RuntimeError):
            ctx.syev_batched([a])
        b = np.eye(n)
        w, _ = ctx.syev_batched([b])
        assert np.array_equal(w[0], np.ones(n))
    finally:
        ctx.close()
