"""The grid barrier of the panel tridiagonalisation is bounded, shown without a
GPU fault: the barriers are told (on the host) to expect one CTA more than is
launched, with the wait bound at 2^14 polls.  Each wait runs out, the launch
ends early, the error comes back as a status, and the same context then solves
the same blocks.  Blocks above 1776 rows take panels for their leading columns;
with NRGB_TRD_PATH=panel all do."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path,sizes", [("panel", [40, 200, 700]), ("", [1850, 300])])
def test_panel_wait_runs_out_and_the_context_stays_usable(monkeypatch, path, sizes):
    import nrgb
    monkeypatch.setenv("NRGB_TRD_PATH", path)
    rng = np.random.default_rng(len(path))
    mats = []
    for n in sizes:
        a = rng.standard_normal((n, n))
        mats.append(a + a.T)
    ctx = nrgb.Context(0)
    try:
        ctx.set_wait_limit(14)
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
