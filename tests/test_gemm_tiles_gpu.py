"""The grouped GEMM's tile sizes and descriptor routes at their edges: 32 x 32
and 64 x 64 tiles, descriptors as kernel parameters (up to 4096 and 32000 bytes)
and through copies, every combination of transposition and 16-byte alignment,
odd leading dimensions and offsets, K remainders, several segments, beta.  The
matrices hold small integers, so every product is exact and must be equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _operand(rng, rows, cols, trans, pad, off):
    """(device buffer, pointer, ld, matrix): op(stored) = matrix, rows x cols."""
    m = rng.integers(-4, 5, (rows, cols)).astype(np.float64)
    stored = m.T if trans else m
    ld = stored.shape[0] + pad
    buf = np.zeros(off + ld * stored.shape[1])
    for j in range(stored.shape[1]):
        buf[off + j * ld:off + j * ld + stored.shape[0]] = stored[:, j]
    t = torch.tensor(buf, device="cuda:0")
    return t, t.data_ptr() + 8 * off, ld, m


def _run(problems, rng):
    import nrgb
    outs, terms, refs, keep = [], [], [], []
    for q, (m, n, ks) in enumerate(problems):
        c0 = rng.integers(-4, 5, (m, n)).astype(np.float64)
        beta = float(q % 3)
        ref = beta * c0
        first = len(terms)
        for s, k in enumerate(ks):
            v = q + s
            ta, tb = v & 1, (v >> 1) & 1
            a, ap, lda, am = _operand(rng, m, k, ta, v % 3, (v >> 2) & 1)
            b, bp, ldb, bm = _operand(rng, k, n, tb, (v + 1) % 3, (v >> 3) & 1)
            alpha = (1.0, -2.0, 0.5)[v % 3]
            terms.append(nrgb.GemmTerm(ap, bp, lda, ldb, k, ta, tb, alpha))
            keep += [a, b]
            ref = ref + alpha * (am @ bm)
        c = torch.tensor(np.ascontiguousarray(c0.T), device="cuda:0")
        outs.append(nrgb.GemmOut(c.data_ptr(), m, m, n, beta, first, len(ks)))
        refs.append((c, ref))
    ctx = nrgb.Context(0)
    try:
        ctx.gemm_grouped_dev(outs, terms)
    finally:
        ctx.close()
    for (c, ref), p in zip(refs, problems):
        assert np.array_equal(c.cpu().numpy().T, ref), p


EDGES = [1, 7, 31, 32, 33, 63, 64, 65, 97, 130]


@pytest.mark.parametrize("name,problems", [
    # a few problems: parameters of 4096 bytes, 32 x 32 tiles
    ("few", [(EDGES[i], EDGES[-1 - i], [1 + 5 * i, 16]) for i in range(10)]),
    # more: parameters of 32000 bytes
    ("many", [(EDGES[i % 10], EDGES[(3 * i + 1) % 10], [15 + i % 4, 33, 1]) for i in range(120)]),
    # beyond: copies
    ("copies", [(EDGES[i % 10], EDGES[(7 * i + 2) % 10], [17, 3 + i % 31]) for i in range(300)]),
    # 64 x 64 tiles, both routes
    ("large", [(600 + q, 601 - q, [100 + q, 31]) for q in range(4)]),
    ("large_copies", [(530 + q % 3, 541, [16, 1, 17]) for q in range(200)]),
    # one short and one long K
    ("long", [(64, 64, [2000]), (33, 65, [1]), (5, 200, [777, 12])]),
])
def test_integer_products_are_exact(name, problems):
    _run(problems, np.random.default_rng(len(name)))


def test_basis_change_without_allocations_is_exact():
    import ctypes as C

    import nrgb
    rng = np.random.default_rng(5)
    for sizes in ([(1, 3), (33, 64), (65, 31), (100, 130)], [(5 + i % 40, 3 + i % 37) for i in range(700)]):
        zb, zk, op, out, refs = [], [], [], [], []
        for i, j in sizes:
            b, k, o = (rng.integers(-3, 4, s).astype(np.float64) for s in ((i, i), (j, j), (i, j)))
            for lst, x in ((zb, b), (zk, k), (op, o)):
                lst.append(torch.tensor(np.ascontiguousarray(x.T), device="cuda:0"))
            out.append(torch.zeros(j, i, dtype=torch.float64, device="cuda:0"))
            refs.append(b.T @ o @ k)
        n = len(sizes)
        ptr = lambda ts: (C.c_void_p * n)(*[t.data_ptr() for t in ts])  # noqa: E731
        rc = nrgb.load().nrgb_basis_change_noalloc(n, (C.c_int * n)(*[s[0] for s in sizes]), (C.c_int * n)(*[s[1] for s in sizes]),
                                                   ptr(zb), ptr(zk), ptr(op), ptr(out), None)
        assert rc == 0
        for t, r in zip(out, refs):
            assert np.array_equal(t.cpu().numpy().T, r)
