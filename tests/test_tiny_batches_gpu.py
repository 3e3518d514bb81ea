"""Blocks up to 32 rows, alone and beside larger ones: calls with few of them
(descriptors as a kernel parameter, up to 96), one more than that and many.

Tolerance: 10 n eps for the residual and the orthogonality of a backward stable
solver, as for the larger blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 95, 96, 97, 300])
@pytest.mark.parametrize("larger", [(), (33, 70)])
def test_many_tiny_blocks(count, larger):
    import nrgb
    rng = np.random.default_rng(count + len(larger))
    ns = [int(rng.integers(1, 33)) for _ in range(count)] + list(larger)
    mats = []
    for n in ns:
        a = rng.standard_normal((n, n))
        mats.append(a + a.T)
    ctx = nrgb.Context(0)
    try:
        ws, zs = ctx.syev_batched(mats)
    finally:
        ctx.close()
    for m, w, z in zip(mats, ws, zs):
        n = len(w)
        tol = 10 * n * 2.0 ** -52
        assert np.all(np.diff(w) >= 0)
        assert np.max(np.abs(z.T @ z - np.eye(n))) <= tol
        assert np.max(np.abs(m @ z - z * w[None, :])) <= tol * max(1.0, np.max(np.abs(m)) * np.sqrt(n))
