"""Grouped products whose launch is reordered by length (more than one wave of
CTAs): every output lands in its place with its own beta and terms, for
descriptors that travel with the launch and for those that do not fit there.

Tolerance: an FP64 product of inner dimension k differs from another order of its
sum by at most 2 k 2^-53 |A| |B|; k <= 330 in all, beta and alpha at most 1."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("count,edge", [(40, 300), (300, 90), (700, 70)])
def test_reordered_launches(count, edge):
    import nrgb
    g = torch.Generator(device="cuda:0").manual_seed(count)
    r = torch.Generator().manual_seed(count)
    rand = lambda *s: torch.randn(*s, dtype=torch.float64, device="cuda:0", generator=g)  # noqa: E731
    outs, terms, keep = [], [], []
    for p in range(count):
        m, n = (int(torch.randint(edge // 2, edge + 1, (1,), generator=r)) for _ in range(2))
        beta = (0.0, 1.0, -0.5)[p % 3]
        c = rand(n, m)
        want, size, t0 = beta * c.T, c.T.abs(), len(terms)
        for q in range(1 + p % 3):
            k, alpha = 1 + int(torch.randint(0, 110, (1,), generator=r)), (1.0, 0.7)[p & 1]
            a, b = rand(k, m), rand(n, k)
            terms.append(nrgb.GemmTerm(a.data_ptr(), b.data_ptr(), m, k, k, 0, 0, alpha))
            want, size = want + alpha * (a.T @ b.T), size + (a.T.abs() @ b.T.abs())
            keep += [a, b]
        outs.append(nrgb.GemmOut(c.data_ptr(), m, m, n, beta, t0, len(terms) - t0))
        keep.append((c, want, size))
    ctx = nrgb.Context(0)
    try:
        ctx.gemm_grouped_dev(outs, terms)
        torch.cuda.synchronize()
    finally:
        ctx.close()
    for c, want, size in (x for x in keep if isinstance(x, tuple)):
        assert bool(torch.all((c.T - want).abs() <= 2 * 332 * 2.0 ** -53 * (size.abs() + 1e-300) + 2.0 ** -50 * size.abs()))
