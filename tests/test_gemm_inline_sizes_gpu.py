"""Grouped products over every size of parameter block that carries their
descriptors (4, 8, 16 and 32 KB; an output and its term are 112 bytes) and
beyond, each launch more than one wave of CTAs and so reordered, with and
without scaling, with 32 x 32 and with 64 x 64 tiles.

Tolerance: an FP64 product of inner dimension k differs from another order of its
sum by at most 2 k 2^-53 |A| |B|; k <= 100, and a rounding for beta C and for
alpha."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("alpha", [1.0, -0.7])
@pytest.mark.parametrize("count,lo,hi", [(30, 130, 192), (60, 66, 128), (100, 66, 128), (250, 66, 100), (400, 40, 90),
                                         (8, 600, 640), (12, 384, 384)])
def test_every_parameter_block(count, lo, hi, alpha):
    import nrgb
    g = torch.Generator(device="cuda:0").manual_seed(count)
    r = torch.Generator().manual_seed(count)
    rand = lambda *s: torch.randn(*s, dtype=torch.float64, device="cuda:0", generator=g)  # noqa: E731
    pick = lambda x, y: int(torch.randint(x, y + 1, (1,), generator=r))  # noqa: E731
    outs, terms, keep = [], [], []
    for p in range(count):
        m, n, k = pick(lo, hi), pick(lo, hi), pick(1, 100)
        beta = (0.0, 1.0, -0.5)[p % 3]
        a, b, c = rand(k, m), rand(n, k), rand(n, m)
        want = beta * c.T + alpha * (a.T @ b.T)
        size = c.T.abs() + a.T.abs() @ b.T.abs()
        terms.append(nrgb.GemmTerm(a.data_ptr(), b.data_ptr(), m, k, k, 0, 0, alpha))
        outs.append(nrgb.GemmOut(c.data_ptr(), m, m, n, beta, p, 1))
        keep.append((a, b, c, want, size))
    ctx = nrgb.Context(0)
    try:
        ctx.gemm_grouped_dev(outs, terms)
        torch.cuda.synchronize()
    finally:
        ctx.close()
    for _, _, c, want, size in keep:
        assert bool(torch.all((c.T - want).abs() <= (2 * 100 + 4) * 2.0 ** -53 * size))
