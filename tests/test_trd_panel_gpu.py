"""The panel tridiagonalisation: blocks beyond the many-CTA kernel (n > 1776,
panels for their leading columns, then the mirrored trailing block), and blocks of
any size with NRGB_TRD_PATH=panel: fewer rows than a tile (64 x 32) or a panel
(32), remainders of both, more CTAs than tiles, several blocks at once.

Tolerance: a backward stable solver leaves a residual and a loss of orthogonality
of a small multiple of n eps; 10 n eps max-norm wise (|A| of a random symmetric
matrix grows as sqrt(n), which is left out on the safe side)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _check(ns, seed):
    import nrgb
    rng = np.random.default_rng(seed)
    mats = []
    for n in ns:
        a = rng.standard_normal((n, n))
        mats.append(a + a.T)
    ctx = nrgb.Context(0)
    try:
        ws, zs = ctx.syev_batched([m.copy() for m in mats])
    finally:
        ctx.close()
    for m, w, z in zip(mats, ws, zs):
        n = len(w)
        A, W = torch.from_numpy(m).cuda(), torch.from_numpy(np.ascontiguousarray(w)).cuda()
        Z = torch.from_numpy(np.ascontiguousarray(z)).cuda()
        tol = 10 * n * 2.0 ** -52
        assert bool(torch.all(W[1:] >= W[:-1]))
        eye = torch.eye(n, dtype=torch.float64, device="cuda:0")
        assert (Z.T @ Z - eye).abs().max().item() <= tol
        res = min((A @ Y - Y * W[None, :]).abs().max().item() for Y in (Z, Z.T))
        assert res <= tol * max(1.0, A.abs().max().item())


@pytest.mark.parametrize("ns", [(33, 34, 64, 65), (95, 96, 97, 129), (257, 300, 40), (800,)])
def test_panels_alone(ns, monkeypatch):
    monkeypatch.setenv("NRGB_TRD_PATH", "panel")
    _check(ns, sum(ns))


@pytest.mark.parametrize("ns", [(1777,), (1808, 1809), (2000, 1900, 300)])
def test_panels_then_many_ctas(ns):
    _check(ns, sum(ns))
