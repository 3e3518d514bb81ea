"""Blocks of low rank: what the first reflectors leave is rounding, then rounding
of rounding, until the squares of a column underflow.  All ones, outer products
and sums of two of them, with the scales and sizes of every tridiagonalisation
path, whole and by panels alone.

Eigenvalues, residual and orthogonality within 1e-13 max(10, n) ||A||, the bound
of the other eigensolver tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMALL = list(range(2, 33))
MEDIUM = list(range(33, 130)) + [200, 300, 301, 464, 512, 640]
LARGE = [641, 700, 1000, 1850]


def _check(sizes, kind):
    import nrgb
    rng = np.random.default_rng(17)
    mats = []
    for n in sizes:
        if kind == "ones":
            mats.append(np.ones((n, n)))
        elif kind == "scaled":
            mats.append(0.7e-3 * np.ones((n, n)))
        elif kind == "outer":
            x = rng.uniform(0.5, 2.0, n)
            mats.append(np.outer(x, x))
        else:
            x, y = rng.choice([-1.0, 1.0, 2.0], n), rng.uniform(-1.0, 1.0, n)
            mats.append(np.outer(x, x) - np.outer(y, y))
    ctx = nrgb.Context(0)
    try:
        ws, zs = ctx.syev_batched(mats)
    finally:
        ctx.close()
    for a, w, z in zip(mats, ws, zs):
        n = a.shape[0]
        ref = np.linalg.eigvalsh(a)
        tol = 1e-13 * max(10, n)
        norm = np.max(np.abs(ref))
        assert np.max(np.abs(w - ref)) <= tol * norm, ("eigenvalues", kind, n)
        assert np.max(np.abs(a @ z - z * w)) <= tol * norm, ("residual", kind, n)
        assert np.max(np.abs(z.T @ z - np.eye(n))) <= tol, ("orthogonality", kind, n)


@pytest.mark.parametrize("kind", ["ones", "scaled", "outer", "two"])
@pytest.mark.parametrize("sizes", [SMALL, MEDIUM, LARGE], ids=["small", "medium", "large"])
def test_low_rank(sizes, kind):
    _check(sizes, kind)


@pytest.mark.parametrize("kind", ["ones", "outer"])
def test_low_rank_by_panels(monkeypatch, kind):
    monkeypatch.setenv("NRGB_TRD_PATH", "panel")
    _check([33, 64, 100, 129, 301, 700], kind)
