"""The digits of the split-precision products where they can go wrong: rows
whose largest entry lies on either side of what D balanced 8-bit digits hold,
rows and columns of very different scales, rows of zeros, inner dimensions
around a chunk (32) and a piece (128) of the slicing passes, and more output
tiles than persistent CTAs, against products in extended precision.

Bound: with D digits a scaled entry's remainder is at most 2^-8D, the D - 1
digit products of the first order left out are at most 2^-8D each (those of
higher orders add less than 1/64 of that), and a row's scale 2^E is at most
2.01 times its largest entry:
k (D + 2) 2.01^2 (1 + 2^-6) 2^-8D max|row| max|column|, below the 4.2 of the
test, and two roundings of the result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _rows(rng, rows, k):
    x = rng.uniform(-1.0, 1.0, (rows, k)) * 2.0 ** rng.integers(-60, 61, (rows, 1))
    edge = [1.0 - 2.0 ** -53, 127.5 / 128, np.nextafter(127.5 / 128, 0), 0x7F7F7F7F7F7F7F / 2.0 ** 55, -127.75 / 128, 0.5]
    for i in range(rows):
        if i % 3 == 0:
            x[i, i % k] = edge[(i // 3) % len(edge)] * 2.0 ** rng.integers(-60, 61)
        elif i % 7 == 1:
            x[i] = 0.0
    return x


@pytest.mark.parametrize("slices", [2, 5, 6, 7, 8])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (129, 63, 31), (64, 65, 33), (127, 130, 127), (128, 64, 128),
                                   (40, 70, 129), (3, 2, 400)])
def test_split_digits_at_edges(slices, m, n, k):
    import nrgb
    rng = np.random.default_rng(1000 * slices + m + n + k)
    A, B = _rows(rng, m, k), _rows(rng, n, k).T
    D = min(slices, 7)
    ref = (A.astype(np.longdouble) @ B.astype(np.longdouble))
    bound = 4.2 * k * (D + 2) * 2.0 ** (-8 * D) * np.abs(A).max(1)[:, None] * np.abs(B).max(0)[None, :]
    ctx = nrgb.Context(0)
    try:
        for ta in (0, 1):
            for tb in (0, 1):
                a = torch.from_numpy(np.ascontiguousarray(A if ta else A.T)).cuda()  # column-major storage
                b = torch.from_numpy(np.ascontiguousarray(B if tb else B.T)).cuda()
                c = torch.full((n, m), 3.0, dtype=torch.float64, device="cuda:0")
                out = nrgb.GemmOut(c.data_ptr(), m, m, n, 0.0, 0, 1)
                term = nrgb.GemmTerm(a.data_ptr(), b.data_ptr(), k if ta else m, n if tb else k, k, ta, tb, 1.0)
                ctx.gemm_grouped_split_dev(slices, [out], [term])
                got = c.cpu().numpy().T
                assert np.all(np.abs(got - ref) <= bound + 2.0 ** -52 * np.abs(ref))
    finally:
        ctx.close()


def test_split_more_tiles_than_ctas():
    """Every CTA takes several tiles of several problems, with two segments."""
    import nrgb
    g = torch.Generator(device="cuda:0").manual_seed(5)
    ctx = nrgb.Context(0)
    try:
        outs, terms, keep = [], [], []
        for m, n in ((700, 900), (130, 2000), (1500, 65), (257, 641)):
            c = torch.randn(n, m, dtype=torch.float64, device="cuda:0", generator=g)
            want, t0 = 0.5 * c.T, len(terms)
            big = torch.zeros(m, n, dtype=torch.float64, device="cuda:0")
            for k, alpha in ((90, 1.0), (37, -0.5)):
                a = torch.randn(k, m, dtype=torch.float64, device="cuda:0", generator=g)
                b = torch.randn(n, k, dtype=torch.float64, device="cuda:0", generator=g)
                terms.append(nrgb.GemmTerm(a.data_ptr(), b.data_ptr(), m, k, k, 0, 0, alpha))
                want = want + alpha * (a.T @ b.T)
                big += k * a.abs().amax(0)[:, None] * b.abs().amax(1)[None, :]
                keep += [a, b]
            outs.append(nrgb.GemmOut(c.data_ptr(), m, m, n, 0.5, t0, 2))
            keep.append((c, want, big))
        ctx.gemm_grouped_split_dev(8, outs, terms)
        for c, want, big in (x for x in keep if isinstance(x, tuple)):
            # the digits' bound (37 of 2^-56) and an FP64 product's own (k 2^-53)
            assert bool(torch.all((c.T - want).abs() <= big * 2.0 ** -50 + 2.0 ** -50))
    finally:
        ctx.close()
