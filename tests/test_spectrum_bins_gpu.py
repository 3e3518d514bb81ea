"""The binning kernels of the spectral functions (nrgb_spectrum_fdm,
nrgb_spectrum_dmnrg) at the sizes where their index stepping and their runs of
equal bins can go wrong: one row or one column, rows around the 256 elements a
pass takes, blocks that span several CTAs, degenerate energies, equal energies
of both blocks (E = 0), energies beyond both ends of the grid, and weights on
both sides of the discard threshold.

Tolerance: a bin sums at most dim1 * dimp = 20100 weights, each a product of
six rounded factors and split over two bins at a position whose logarithm
carries about 4 ulp, times 10 bins a decade over 8 decades; the sums of
absolute weights bound the error by (20100 + 6 + 4 * 80) * 2^-53, below 3e-12."""
import numpy as np
import pytest

import nrg_oracle as O

pytestmark = pytest.mark.gpu

BPD, EMIN, EMAX, DISCARD = 10, 1e-5, 1.0, 1e-6
GRID = {"bins": BPD, "emin": EMIN, "emax": EMAX, "discard_immediately": DISCARD}
SHAPES = [(1, 1), (1, 300), (300, 1), (255, 5), (256, 33), (257, 31), (100, 201), (7, 600)]


def _energies(rng, n):
    """Ascending, with runs of equal values and values of the other block."""
    e = np.round(10.0 ** rng.uniform(-7.0, 1.5, n), 6)
    e[n // 3:n // 2] = 0.25
    return np.sort(e)


def _close(got, cs, ab):
    for g, w, s in ((got[0], cs.pos.w, ab.pos.w), (got[1], cs.neg.w, ab.neg.w)):
        assert g.shape == w.shape
        assert np.all(np.abs(g - w) <= 3e-12 * np.max(s) + 1e-300)


def _add(cs, ab, e, w):
    e, w = np.ravel(e), np.ravel(w)
    keep = ~(np.abs(w) < DISCARD * np.abs(e))
    cs.add(e[keep], w[keep])
    ab.add(e[keep], np.abs(w[keep]))


@pytest.mark.parametrize("allj,alli", SHAPES)
def test_fdm_bins_at_edges(allj, alli):
    import nrgb
    rng = np.random.default_rng(allj * 1000 + alli)
    T, wn, sf = 0.4, 0.37, 1.3
    retj, reti = allj // 2, (2 * alli) // 3
    Ej, Ei = _energies(rng, allj), _energies(rng, alli)
    A, B = rng.standard_normal((2, allj, alli)) * 10.0 ** rng.uniform(-5, 0, (2, allj, alli))
    rj, ri = rng.standard_normal((retj, retj)), rng.standard_normal((reti, reti))
    ctx = nrgb.Context(0)
    try:
        up = ctx.mat_upload
        pair = nrgb.FdmPair(up(A), up(B), up(ri) if reti else -1, up(rj) if retj else -1, up(Ei[None, :]),
                            up(Ej[None, :]), reti, retj, sf)
        got = ctx.spectrum_fdm([pair], T, wn, 1, BPD, EMIN, EMAX, DISCARD)
    finally:
        ctx.close()
    cs, ab = O.ChainSpectrum(GRID, 10), O.ChainSpectrum(GRID, 10)
    dE = Ej[:, None] - Ei[None, :]
    wg = sf * A * B * wn * np.exp(-Ei / T)[None, :]
    wl = sf * A * B * wn * np.exp(-Ej / T)[:, None]
    _add(cs, ab, dE[:, reti:], wg[:, reti:])
    _add(cs, ab, dE[retj:, :reti], sf * A[retj:, :reti] * (B[:, :reti] @ ri)[retj:, :])
    _add(cs, ab, dE[retj:, :], wl[retj:, :])
    _add(cs, ab, dE[:retj, reti:], sf * A[:retj, reti:] * (rj @ B[:retj, :])[:, reti:])
    _close(got, cs, ab)


@pytest.mark.parametrize("dim1,dimp", SHAPES)
def test_dmnrg_bins_at_edges(dim1, dimp):
    import nrgb
    rng = np.random.default_rng(dim1 * 1000 + dimp)
    scale, wmin, wmax, sf = 0.3, 1e-4, 8.0, 0.7
    E1, Ep = _energies(rng, dim1), _energies(rng, dimp)
    A, B = rng.standard_normal((2, dim1, dimp)) * 10.0 ** rng.uniform(-5, 0, (2, dim1, dimp))
    r1, rp = rng.standard_normal((dim1, dim1)), rng.standard_normal((dimp, dimp))
    ctx = nrgb.Context(0)
    try:
        up = ctx.mat_upload
        pair = nrgb.DmnrgPair(up(A), up(B), up(r1), up(rp), up(E1[None, :]), up(Ep[None, :]), sf)
        got = ctx.spectrum_dmnrg([pair], scale, wmin, wmax, 1, BPD, EMIN, EMAX, DISCARD)
    finally:
        ctx.close()
    cs, ab = O.ChainSpectrum(GRID, 10), O.ChainSpectrum(GRID, 10)
    dE = E1[:, None] - Ep[None, :]
    w = sf * ((B @ rp) * A + (r1 @ A) * B)
    on = ~((np.abs(dE) < wmin) | (np.abs(dE) > wmax))
    _add(cs, ab, scale * dE[on], w[on])
    _close(got, cs, ab)
