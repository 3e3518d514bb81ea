"""The cluster tridiagonalisation at the edges of its shapes: sizes on both
sides of every row and cluster limit, whole blocks and the trailing part of
larger ones, matrices whose columns need no reflector, all against LAPACK
(eigenvalues, residual and orthogonality within 1e-13 n ||A||, the bound of
the other eigensolver tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [33, 63, 64, 65, 96, 97, 128, 129, 160, 161, 192, 193, 224, 225, 256, 257, 288, 289, 320, 321, 384, 385, 448,
         449, 480, 481, 512, 513, 576, 577, 640, 641, 672, 700]


def _matrices(kind, rng):
    out = []
    for n in SIZES:
        a = rng.standard_normal((n, n))
        a = a + a.T
        if kind == "decoupled":  # every third row and column zero off the diagonal: reflectors of zero columns
            a[::3, :] = 0.0
            a[:, ::3] = 0.0
            a[np.arange(n), np.arange(n)] = rng.standard_normal(n)
        elif kind == "diagonal":
            a = np.diag(rng.standard_normal(n))
        elif kind == "graded":
            s = np.logspace(0, -6, n)
            a = a * s[:, None] * s[None, :]
        out.append(a)
    return out


@pytest.mark.parametrize("kind", ["gaussian", "decoupled", "diagonal", "graded"])
def test_every_shape_against_lapack(kind):
    import nrgb
    mats = _matrices(kind, np.random.default_rng(len(kind)))
    ctx = nrgb.Context(0)
    try:
        ws, zs = ctx.syev_batched(mats)
    finally:
        ctx.close()
    for a, w, z in zip(mats, ws, zs):
        n = a.shape[0]
        tol = 1e-13 * n * max(np.linalg.norm(a, 2), 1e-300)
        assert np.max(np.abs(w - np.linalg.eigvalsh(a))) <= tol, ("eigenvalues", kind, n)
        assert np.max(np.abs(a @ z - z * w)) <= tol, ("residual", kind, n)
        assert np.max(np.abs(z.T @ z - np.eye(n))) <= 1e-13 * n, ("orthogonality", kind, n)
