"""The tridiagonalisation kernels that hold the matrix in registers (a cluster
per block; many CTAs per block beyond) at the edges of their shapes: sizes on
both sides of every row and CTA limit, whole blocks and the trailing part of
larger ones, matrices whose columns need no reflector, all against LAPACK
(eigenvalues, residual and orthogonality within 1e-13 n ||A||, the bound of
the other eigensolver tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [33, 63, 64, 65, 96, 97, 128, 129, 160, 161, 192, 193, 224, 225, 256, 257, 288, 289, 320, 321, 384, 385, 448,
         449, 480, 481, 512, 513, 576, 577, 640]
LARGE = [641, 768, 769, 896, 897, 1024, 1025, 1280, 1281, 1500, 1536, 1537, 1776, 1777, 1850]


def _matrices(kind, rng, sizes):
    out = []
    for n in sizes:
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


@pytest.mark.parametrize("kind,sizes", [("gaussian", SIZES), ("decoupled", SIZES), ("diagonal", SIZES),
                                        ("graded", SIZES), ("gaussian", LARGE), ("decoupled", LARGE[1::4]),
                                        ("diagonal", LARGE[2::4])])
def test_every_shape_against_lapack(kind, sizes):
    import nrgb
    mats = _matrices(kind, np.random.default_rng(len(kind)), sizes)
    ctx = nrgb.Context(0)
    try:
        ws, zs = ctx.syev_batched(mats)
    finally:
        ctx.close()
    for a, w, z in zip(mats, ws, zs):
        n = a.shape[0]
        ref = np.linalg.eigvalsh(a)
        tol = 1e-13 * n * np.max(np.abs(ref))
        assert np.max(np.abs(w - ref)) <= tol, ("eigenvalues", kind, n)
        assert np.max(np.abs(a @ z - z * w)) <= tol, ("residual", kind, n)
        assert np.max(np.abs(z.T @ z - np.eye(n))) <= 1e-13 * n, ("orthogonality", kind, n)
