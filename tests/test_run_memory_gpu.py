"""Device memory of a run is given back at its end: what the context still
holds of the device's default memory pool is less than one chunk of the run's
slabs (1 MiB; the truncation's arrays, which the next run replaces, are tens of
kilobytes for a run this small)."""
import ctypes
import os

import pytest

import inputgen

pytestmark = pytest.mark.gpu


def _pool_used():
    """Bytes allocated from device 0's default memory pool."""
    cu = ctypes.CDLL("libcuda.so.1")
    assert cu.cuInit(0) == 0
    dev, pool, used = ctypes.c_int(), ctypes.c_void_p(), ctypes.c_uint64()
    assert cu.cuDeviceGet(ctypes.byref(dev), 0) == 0
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), dev) == 0
    assert cu.cuMemPoolGetAttribute(pool, 7, ctypes.byref(used)) == 0  # CU_MEMPOOL_ATTR_USED_MEM_CURRENT
    return used.value


def test_a_finished_run_holds_no_chunks(tmp_path):
    import nrgb
    wd, od = str(tmp_path / "in"), str(tmp_path / "out")
    inputgen.make_siam(wd, 0.2, -0.05, 0.02, 2.0, 12,
                       params={"keep": 60, "fdm": True, "T": 1e-3, "specd": "A_d-A_d", "bins": 20, "savebins": True,
                               "broaden": False})
    os.makedirs(od)
    ctx = nrgb.Context(0)
    try:
        before = _pool_used()
        for _ in range(2):
            ctx.run(wd, od)
            assert _pool_used() - before < 1 << 20
    finally:
        ctx.close()
