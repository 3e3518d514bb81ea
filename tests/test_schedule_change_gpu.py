"""Another thread changes the schedule's cluster limit while the solver plans
its calls: a call takes one value of the limit for all of its decisions (the
exchange buffers of the many-CTA tridiagonalisation among them), so every call
solves its blocks."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_limit_changes_during_calls():
    import nrgb
    rng = np.random.default_rng(8)
    mats = []
    for n in (41, 100, 301, 500):
        a = rng.standard_normal((n, n))
        mats.append(a + a.T)
    refs = [np.linalg.eigvalsh(a) for a in mats]
    ctx, other = nrgb.Context(0), nrgb.Context(0)
    saved = ctx.get_schedule()
    stop = threading.Event()

    def change():
        k = 0
        while not stop.is_set():
            other.set_schedule((0, 40)[k & 1], saved["gemm_large_from"])
            k += 1

    th = threading.Thread(target=change)
    th.start()
    try:
        for _ in range(100):
            ws, _ = ctx.syev_batched(mats)
            for a, w, ref in zip(mats, ws, refs):
                assert np.max(np.abs(w - ref)) <= 1e-13 * len(ref) * np.max(np.abs(ref))
    finally:
        stop.set()
        th.join()
        ctx.set_schedule(saved["cluster_limit"], saved["gemm_large_from"])
        other.close()
        ctx.close()
