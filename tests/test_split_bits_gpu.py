"""Split-precision products of entries near the top of a binade, where the
balanced digits of a row need the next power of two as its scale: the error
stays below the documented bound k 2^-7S (S + 3) max|row| max|column|.

The entry x = y 2^-54 has the balanced digits (64, -63, -128, -128, ...): a
product of two of them has digit products of one sign and nearly the largest
size in every order, so whatever an implementation leaves out adds up.  Seven
digits for 8 slices leave out the products of the order 2^-56, 19.9 k 2^-56 of
the largest entries' product here; the bound is 11 k 2^-56.  The exact product
is formed with integers."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

Y = (64 << 48) - (63 << 40) - sum(128 << (8 * i) for i in range(5))


@pytest.mark.parametrize("slices", [2, 4, 7, 8])
@pytest.mark.parametrize("k", [1, 31, 64, 500])
def test_rows_that_take_the_next_scale(slices, k):
    import nrgb
    x = float(Y) * 2.0 ** -54
    assert int(x * 2.0 ** 54) == Y and x > 127.4981 / 128
    m, n = 130, 65
    ra, cb = 2.0 ** (np.arange(m) % 37 - 18), 2.0 ** (np.arange(n) % 29 - 14)
    A, B = np.outer(ra, np.full(k, x)), np.outer(np.full(k, x), cb)
    exact = k * Fraction(Y, 1 << 54) ** 2
    ctx = nrgb.Context(0)
    try:
        for ta in (0, 1):
            for tb in (0, 1):
                a = torch.from_numpy(np.ascontiguousarray(A if ta else A.T)).cuda()  # column-major storage
                b = torch.from_numpy(np.ascontiguousarray(B if tb else B.T)).cuda()
                c = torch.zeros((n, m), dtype=torch.float64, device="cuda:0")
                out = nrgb.GemmOut(c.data_ptr(), m, m, n, 0.0, 0, 1)
                term = nrgb.GemmTerm(a.data_ptr(), b.data_ptr(), k if ta else m, n if tb else k, k, ta, tb, 1.0)
                ctx.gemm_grouped_split_dev(slices, [out], [term])
                got = c.cpu().numpy().T / np.outer(ra, cb)  # powers of two: exact
                worst = max(abs(Fraction(float(g)) - exact) for g in np.unique(got))
                assert worst <= Fraction(k * (slices + 3), 1 << (7 * slices)) * Fraction(x) ** 2, (ta, tb)
    finally:
        ctx.close()
