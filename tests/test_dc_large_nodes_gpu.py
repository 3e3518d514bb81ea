"""Merges of more than 5600 rows, whose deflation scan works in global memory
instead of shared memory: one block with single and one with fourfold
eigenvalues (rotations of close pairs).  Residual and orthogonality within
1e-13 n ||A||, the bound of the other eigensolver tests, and the trace."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

N = 5640  # the last merge has N rows, the two before it half as many


@pytest.mark.parametrize("kind", ["gaussian", "fourfold"])
def test_merge_beyond_shared_memory(kind):
    import nrgb
    g = torch.Generator(device="cuda:0").manual_seed(7)
    a = torch.randn(N, N, dtype=torch.float64, device="cuda:0", generator=g)
    if kind == "fourfold":
        q, _ = torch.linalg.qr(a)
        lam = torch.randn(N // 4, dtype=torch.float64, device="cuda:0", generator=g).repeat_interleave(4)
        a = (q * lam) @ q.T
    a = a + a.T
    ctx = nrgb.Context(0)
    try:
        (w,), (z,) = ctx.syev_batched([a.cpu().numpy()])
    finally:
        ctx.close()
    assert np.all(np.diff(w) >= 0)
    w, z = torch.from_numpy(np.ascontiguousarray(w)).cuda(), torch.from_numpy(np.ascontiguousarray(z)).cuda()
    tol = 1e-13 * N * w.abs().max()
    assert (a @ z - z * w).abs().max() <= tol
    assert (z.T @ z - torch.eye(N, dtype=torch.float64, device="cuda:0")).abs().max() <= 1e-13 * N
    assert (w.sum() - a.diagonal().sum()).abs() <= tol
