"""The waits inside a cluster of the register tridiagonalisation are bounded,
shown without a GPU fault: the waits are told (on the host) to expect one word
more than the cluster's CTAs send, with their bound at 2^12 tries.  Each wait
runs out, the CTAs stop sending and end together, the error comes back as a
status, and the same context then solves the same blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_cluster_wait_runs_out_and_the_context_stays_usable():
    import nrgb
    rng = np.random.default_rng(12)
    mats = []
    for n in (65, 200, 301, 500, 640, 64, 20):  # clusters of 2 to 16 CTAs; two without an exchange
        a = rng.standard_normal((n, n))
        mats.append(a + a.T)
    ctx = nrgb.Context(0)
    try:
        ctx.set_wait_limit(12)
        ctx.inject_barrier_shortfall(True)
        with pytest.raises(RuntimeError, match="grid barrier timed out"):
            ctx.syev_batched(mats)
        ctx.inject_barrier_shortfall(False)
        ctx.set_wait_limit(23)
        ws, zs = ctx.syev_batched(mats)
    finally:
        ctx.close()
    for a, w, z in zip(mats, ws, zs):
        n = a.shape[0]
        ref = np.linalg.eigvalsh(a)
        tol = 1e-13 * max(10, n) * np.max(np.abs(ref))
        assert np.max(np.abs(w - ref)) <= tol
        assert np.max(np.abs(a @ z - z * w)) <= tol
