"""The eigensolver's range: matrices scaled by powers of two between about
1e-140 and 1e140 on every tridiagonalisation path (one CTA, one CTA of
registers, clusters, many CTAs, panels), and a column of couplings so small
that the square of its reflector's scale is beyond the largest number while
the square of its norm is still exact to 15 digits.

The reference is LAPACK on the unscaled matrix (a power of two scales
eigenvalues exactly); eigenvalues, residual and orthogonality within 1e-13 n
||A||, the bound of the other eigensolver tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [32, 33, 64, 65, 301, 640, 641, 1850]


def _check(mats, unscaled, scale):
    import nrgb
    ctx = nrgb.Context(0)
    try:
        ws, zs = ctx.syev_batched(mats)
    finally:
        ctx.close()
    for a, w, z in zip(unscaled, ws, zs):
        n = a.shape[0]
        w = np.asarray(w) / scale
        ref = np.linalg.eigvalsh(a)
        tol = 1e-13 * n * np.max(np.abs(ref))
        assert np.max(np.abs(w - ref)) <= tol, ("eigenvalues", n)
        assert np.max(np.abs(a @ z - z * w)) <= tol, ("residual", n)
        assert np.max(np.abs(z.T @ z - np.eye(n))) <= 1e-13 * n, ("orthogonality", n)


@pytest.mark.parametrize("power", [-465, -365, -345, 0, 345, 365, 465])
def test_scaled_matrices(power):
    rng = np.random.default_rng(3)
    mats = [(lambda a: a + a.T)(rng.standard_normal((n, n))) for n in SIZES]
    scale = 2.0 ** power
    _check([a * scale for a in mats], mats, scale)


def test_tiny_couplings_in_a_matrix_of_order_one():
    rng = np.random.default_rng(4)
    mats = []
    for n in SIZES:
        a = rng.standard_normal((n, n))
        a = a + a.T
        a[0, 1:] = np.sqrt(1.3e-309 / n) * rng.choice([-1.0, 1.0], n - 1)
        a[0, 1] = 0.0
        a[1:, 0] = a[0, 1:]
        mats.append(a)
    _check(mats, mats, 1.0)
