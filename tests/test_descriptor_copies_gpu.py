"""Descriptors of a run's grouped products that do not travel as a kernel
parameter go through the run's own (pinned) upload path and count in its
host-to-device bytes: forced for every launch by a schedule that considers
128 x 128 tiles, from an edge that no product reaches."""
import os

import numpy as np
import pytest

import inputgen
import nrg_cases as cases

pytestmark = pytest.mark.gpu


def test_descriptor_copies_are_the_runs_own(tmp_path):
    import nrgb
    wd = str(tmp_path / "in")
    inputgen.make_siam(wd, 0.2, -0.05, 0.02, 2.0, 12,
                       params={"keep": 60, "fdm": True, "T": 1e-3, "specd": "A_d-A_d", "bins": 20, "savebins": True,
                               "broaden": False})
    ctx = nrgb.Context(0)
    saved = ctx.get_schedule()
    h2d, td = [], []
    try:
        for large_from in (0, 1 << 30):
            od = str(tmp_path / ("out%d" % large_from))
            os.makedirs(od)
            ctx.set_schedule(saved["cluster_limit"], large_from)
            st = ctx.run(wd, od)
            h2d.append(st["h2d_bytes"])
            td.append(cases.read_table(os.path.join(od, "td")))
    finally:
        ctx.set_schedule(saved["cluster_limit"], saved["gemm_large_from"])
        ctx.close()
    # every step of both sweeps has products; one problem and one term are 112 bytes
    assert h2d[1] - h2d[0] >= 2 * 11 * 112, h2d
    # the same kernels on the same numbers
    assert np.array_equal(td[0], td[1])
