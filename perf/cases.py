"""What a user of this framework has it do, as cases that can be timed.

Every case goes through the package's public entry points (nrgb.Context,
nrgb.Server and the C functions of include/nrgb.h), from the smallest calls
(one first-iteration step of tiny blocks) to whole NRG runs.  All arithmetic is
FP64; the split-precision products are an option of their own entry point.

listed() gives the standing cases, draw(rng) one more of the same ranges,
prepare(case, seed) what a program holds before the call (device buffers, plan
handles, run directories), run(state) one pass, work(case) the bytes and flops
a pass cannot do without, exact(case, seed) its outputs from plain FP64
torch/numpy where there are such values.

Eigenvectors are unique up to their sign.  As a program that stores or compares
them would, the passes that return eigenvectors (or matrix elements between
them) fix the sign: a fixed random combination of 16 components of each vector
is made positive.
"""
import ctypes
import math
import os
import random
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nrgljubljana-old_b200"))
import inputgen  # noqa: E402
import nrgb  # noqa: E402

DEV = "cuda:0"
F64 = torch.float64
PROBES = 16  # components of an eigenvector that fix its sign


def listed():
    return [
        # the first iterations of a run: a dozen invariant subspaces of a few
        # states each, where launches and latency are all there is
        {"name": "eig_first", "kind": "eig", "blocks": 14, "lo": 1, "hi": 30, "shape": 1},
        # one dsyev call of a host program replaced one for one (host arrays)
        {"name": "dsyev_host", "kind": "dsyev", "n": 301},
        # all blocks of a step of a single-channel run with Nkeep = 1000
        {"name": "eig_keep1000", "kind": "eig", "blocks": 36, "lo": 20, "hi": 464, "shape": 2},
        # a step with large blocks among small ones (two-channel runs with
        # thousands of kept multiplets; the batched-eigensolve benchmark)
        {"name": "eig_wide", "kind": "eig", "blocks": 20, "lo": 48, "hi": 3600, "shape": 3},
        # eigensolve and basis change of operator blocks in one call
        {"name": "eig_recalc", "kind": "eig_recalc", "blocks": 16, "lo": 16, "hi": 1024, "ops": 2, "shape": 4},
        # second stage of a recalculation: ragged sub-blocks of eigenvector
        # matrices, odd leading dimensions, four terms to an output
        {"name": "gemm_recalc", "kind": "gemm", "form": "recalc", "outs": 64, "lo": 61, "hi": 463, "shape": 5},
        # products of large blocks in every transposition
        {"name": "gemm_dense", "kind": "gemm", "form": "dense", "outs": 8, "lo": 900, "hi": 1500, "shape": 6},
        # the split-precision form of the same (8 INT8 slices: FP64 level)
        {"name": "split_dense", "kind": "split", "slices": 8, "outs": 8, "lo": 900, "hi": 1500, "shape": 7},
        # basis change without allocations, operators of a small run
        {"name": "noalloc", "kind": "noalloc", "ops": 40, "lo": 12, "hi": 130, "shape": 8},
        # one step through the step-level plan: assembly, eigensolve and
        # truncation, recalculation, density matrix back, FDM spectral weights
        {"name": "step_plan", "kind": "step", "ancestors": 18, "keep": 1000, "shape": 9},
        # a whole run: SIAM, QS, FDM spectral function of the impurity level
        {"name": "run_siam", "kind": "run", "keep": 1000, "nmax": 40, "z": 0.625, "spectra": "fdm"},
        # the run server with a z-averaging stream: requests of mixed Nkeep
        {"name": "served", "kind": "served", "keeps": "200 500 1000 200 2000 500 1000 200", "nmax": 40, "z": 0.375},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["eig", "eig", "eig", "dsyev", "eig_recalc", "gemm", "gemm", "split", "noalloc", "step", "run", "served"])
    shape = rng.randrange(1 << 20)
    if kind == "eig":
        hi = log_int(8, 3000)
        return {"kind": kind, "blocks": max(2, min(log_int(3, 48), 6_000_000_000 // hi ** 3)), "lo": max(1, hi // log_int(2, 40)),
                "hi": hi, "shape": shape}
    if kind == "dsyev":
        return {"kind": kind, "n": log_int(3, 1200)}
    if kind == "eig_recalc":
        hi = log_int(24, 1100)
        return {"kind": kind, "blocks": rng.randint(3, 16), "lo": max(2, hi // log_int(2, 40)), "hi": hi,
                "ops": rng.randint(1, 4), "shape": shape}
    if kind == "gemm":
        form = rng.choice(["recalc", "dense"])
        hi = log_int(20, 700) if form == "recalc" else log_int(20, 2000)
        return {"kind": kind, "form": form, "outs": rng.randint(3, 80) if hi < 600 else rng.randint(2, 8),
                "lo": max(3, hi // log_int(2, 12)), "hi": hi, "shape": shape}
    if kind == "split":
        hi = log_int(100, 1800)
        return {"kind": kind, "slices": rng.choice([6, 7, 8]), "outs": rng.randint(2, 12), "lo": hi // 2, "hi": hi, "shape": shape}
    if kind == "noalloc":
        hi = log_int(10, 250)
        return {"kind": kind, "ops": rng.randint(2, 50), "lo": max(2, hi // log_int(2, 10)), "hi": hi, "shape": shape}
    if kind == "step":
        return {"kind": kind, "ancestors": rng.randint(6, 24), "keep": log_int(100, 1800), "shape": shape}
    if kind == "run":
        return {"kind": kind, "keep": log_int(80, 1000), "nmax": rng.randint(12, 40), "z": rng.randint(1, 8) / 8,
                "spectra": rng.choice(["fdm", "dmnrg"])}
    return {"kind": kind, "keeps": " ".join(str(rng.choice([200, 500, 1000])) for _ in range(rng.randint(2, 8))),
            "nmax": rng.randint(20, 40), "z": rng.randint(1, 8) / 8}


# ---------------------------------------------------------------------------
# shared pieces
# ---------------------------------------------------------------------------
_kept = {}


def _context():
    if "ctx" not in _kept:
        _kept["ctx"] = nrgb.Context(0)
    return _kept["ctx"]


def _server():
    if "srv" not in _kept:
        _kept["srv"] = nrgb.Server(0, max_runs=8)
    return _kept["srv"]


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _sizes(count, lo, hi, shape):
    """`count` sizes log-uniform in [lo, hi], the largest one hi."""
    r = random.Random(shape)
    return [hi] + [min(hi, int(lo * (hi / lo) ** r.random() + 0.5)) for _ in range(count - 1)]


def _layout(counts):
    """Offsets of arrays of `counts` doubles in one buffer, each on 256 bytes, and the total."""
    off, at = [], 0
    for n in counts:
        off.append(at)
        at += (n + 31) // 32 * 32
    return off, at


def _block(n, g):
    """A block Hamiltonian: the levels of its ancestors on the diagonal, couplings all over it."""
    a = torch.randn(n, n, device=DEV, dtype=F64, generator=g) / math.sqrt(2.0 * n)
    a = a + a.t()
    a.diagonal().add_(torch.rand(n, device=DEV, dtype=F64, generator=g).mul_(8.0).sort().values)
    return a


class _Signs:
    """Signs of the eigenvectors of a list of blocks packed in one buffer (see the module text)."""

    def __init__(self, ns, off, total):
        g = torch.Generator()
        g.manual_seed(77)
        self.coef = torch.randn(PROBES, generator=g, dtype=F64).to(DEV)
        probe, lens, self.first = [], [], []
        for n, o in zip(ns, off):
            self.first.append(len(lens))
            rows = torch.randint(0, n, (n, PROBES), generator=g)
            probe.append(o + torch.arange(n)[:, None] * n + rows)
            lens += [n] * n
            if (pad := (n * n + 31) // 32 * 32 - n * n):
                probe.append(torch.full((1, PROBES), o + n * n))
                lens.append(pad)
        self.probe = torch.cat(probe).to(DEV)
        ids = torch.arange(len(lens), dtype=torch.int32)
        self.column = torch.repeat_interleave(ids, torch.tensor(lens)).to(DEV)
        assert self.column.numel() == total

    def of(self, z):
        s = torch.mv(z[self.probe], self.coef)
        return torch.where(s < 0, -1.0, 1.0).to(F64)

    def fix(self, z, s):
        return z.mul_(s.index_select(0, self.column))


# ---------------------------------------------------------------------------
# batched eigensolver on device memory
# ---------------------------------------------------------------------------
def _eig_prepare(case, seed):
    ns = _sizes(case["blocks"], case["lo"], case["hi"], case["shape"])
    off, total = _layout([n * n for n in ns])
    woff, wtotal = _layout(ns)
    g = _gen(seed)
    h = torch.zeros(total, device=DEV, dtype=F64)
    for n, o in zip(ns, off):
        h[o:o + n * n] = _block(n, g).reshape(-1)
    st = {"ns": ns, "off": off, "woff": woff, "h": h, "a": torch.empty_like(h), "z": torch.zeros_like(h),
          "w": torch.zeros(wtotal, device=DEV, dtype=F64), "signs": _Signs(ns, off, total)}
    for k, o in (("a", off), ("z", off), ("w", woff)):
        st[k + "p"] = [st[k].data_ptr() + 8 * x for x in o]
    return st


def _eig_run(st):
    st["a"].copy_(st["h"])  # the solver destroys its input
    _context().syev_batched_dev(st["ns"], st["ap"], st["wp"], st["zp"], _stream())
    s = st["signs"]
    return {"w": st["w"], "z": s.fix(st["z"], s.of(st["z"]))}


def _eigh_into(st):
    for n, o, wo in zip(st["ns"], st["off"], st["woff"]):
        w, v = torch.linalg.eigh(st["h"][o:o + n * n].view(n, n))
        st["w"][wo:wo + n] = w
        st["z"][o:o + n * n] = v.t().reshape(-1)


def _eig_exact(case, seed):
    st = _eig_prepare(case, seed)
    _eigh_into(st)
    s = st["signs"]
    return {"w": st["w"], "z": s.fix(st["z"], s.of(st["z"]))}


def _eig_work(ns):
    return {"bytes": sum(8.0 * (2 * n * n + n) for n in ns), "flops": sum(14.0 / 3.0 * n ** 3 for n in ns)}


# ---------------------------------------------------------------------------
# one dsyev call on host arrays
# ---------------------------------------------------------------------------
def _dsyev_prepare(case, seed):
    n = case["n"]
    r = np.random.default_rng(5)
    return {"a": np.asfortranarray(_block(n, _gen(seed)).cpu().numpy()), "rows": r.integers(0, n, PROBES),
            "coef": r.standard_normal(PROBES)}


def _dsyev_fix(st, w, z):
    return {"w": w, "z": z * np.where(st["coef"] @ z[st["rows"]] < 0, -1.0, 1.0)}


def _dsyev_run(st):
    w, z = _context().syev_batched([st["a"]])
    return _dsyev_fix(st, w[0], z[0])


def _dsyev_exact(case, seed):
    st = _dsyev_prepare(case, seed)
    return _dsyev_fix(st, *np.linalg.eigh(st["a"]))


# ---------------------------------------------------------------------------
# eigensolve + basis change of operator blocks
# ---------------------------------------------------------------------------
def _eig_recalc_prepare(case, seed):
    st = _eig_prepare(case, seed)
    ns = st["ns"]
    pairs = [(b, (b + 1) % len(ns)) for b in range(len(ns)) for _ in range(case["ops"])]
    off, total = _layout([ns[i] * ns[j] for i, j in pairs])
    st["bra"], st["ket"] = [p[0] for p in pairs], [p[1] for p in pairs]
    st["ooff"] = off
    st["op"] = torch.randn(total, device=DEV, dtype=F64, generator=_gen(seed + 1))
    st["out"] = torch.zeros(total, device=DEV, dtype=F64)
    row = torch.zeros(total, device=DEV, dtype=torch.int32)
    col = torch.zeros(total, device=DEV, dtype=torch.int32)
    for (i, j), o in zip(pairs, off):
        m = ns[i] * ns[j]
        at = torch.arange(m, device=DEV, dtype=torch.int32)
        row[o:o + m] = st["signs"].first[i] + at % ns[i]
        col[o:o + m] = st["signs"].first[j] + at // ns[i]
    st["row"], st["col"] = row, col
    st["opp"] = [st["op"].data_ptr() + 8 * o for o in off]
    st["outp"] = [st["out"].data_ptr() + 8 * o for o in off]
    return st


def _eig_recalc_outputs(st):
    s = st["signs"].of(st["z"])
    st["out"].mul_(s.index_select(0, st["row"])).mul_(s.index_select(0, st["col"]))
    return {"w": st["w"], "op": st["out"]}


def _eig_recalc_run(st):
    st["a"].copy_(st["h"])
    _context().eig_recalc_step_dev(st["ns"], st["ap"], st["wp"], st["zp"], st["bra"], st["ket"], st["opp"], st["outp"],
                                   _stream())
    return _eig_recalc_outputs(st)


def _eig_recalc_exact(case, seed):
    st = _eig_recalc_prepare(case, seed)
    _eigh_into(st)
    ns = st["ns"]
    z = [st["z"][o:o + n * n].view(n, n).t() for n, o in zip(ns, st["off"])]
    for i, j, o in zip(st["bra"], st["ket"], st["ooff"]):
        m = ns[i] * ns[j]
        op = st["op"][o:o + m].view(ns[j], ns[i]).t()
        st["out"][o:o + m] = (z[i].t() @ op @ z[j]).t().reshape(-1)
    return _eig_recalc_outputs(st)


def _eig_recalc_work(case):
    ns = _sizes(case["blocks"], case["lo"], case["hi"], case["shape"])
    w = _eig_work(ns)
    for b, n in enumerate(ns):
        m = ns[(b + 1) % len(ns)]
        w["bytes"] += case["ops"] * 16.0 * n * m
        w["flops"] += case["ops"] * 2.0 * n * m * (n + m)
    return w


# ---------------------------------------------------------------------------
# grouped GEMM, FP64 and split precision
# ---------------------------------------------------------------------------
def _gemm_shapes(case):
    """Per output (m, n, terms); a term is (k, transpose A, transpose B, rows of A's and B's storage, row offsets, alpha)."""
    r = random.Random(case["shape"])
    sizes = _sizes(2 * case["outs"], case["lo"], case["hi"], case["shape"])
    outs = []
    for o in range(case["outs"]):
        m, n = sizes[2 * o], sizes[2 * o + 1]
        terms = []
        if case.get("form") == "recalc":
            for at in range(4):  # Z1[off : off + k, :m]^T T, four ancestors of the block
                k = max(1, m // 4)
                terms.append((k, 1, 0, m, k, at * k if (at + 1) * k <= m else 0, 0, r.uniform(0.5, 1.5)))
        else:
            k = min(case["hi"], int(case["lo"] * (case["hi"] / case["lo"]) ** r.random() + 0.5))
            ta, tb = o & 1, (o >> 1) & 1
            terms.append((k, ta, tb, k if ta else m, n if tb else k, 0, 0, 1.0))
        outs.append((m, n, terms))
    return outs


def _gemm_prepare(case, seed):
    g = _gen(seed)
    st = {"outs": [], "terms": [], "keep": [], "c": [], "slices": case.get("slices", 0)}
    shapes = _gemm_shapes(case)
    off, total = _layout([m * n for m, n, _ in shapes])
    st["out"] = torch.zeros(total, device=DEV, dtype=F64)
    for (m, n, terms), o in zip(shapes, off):
        first = len(st["terms"])
        for k, ta, tb, lda, ldb, oa, ob, alpha in terms:
            a = torch.randn(m if ta else k, lda, device=DEV, dtype=F64, generator=g)  # column-major lda x columns
            b = torch.randn(k if tb else n, ldb, device=DEV, dtype=F64, generator=g)
            st["keep"].append((a, b, k, ta, tb, oa, ob, alpha))
            st["terms"].append(nrgb.GemmTerm(a.data_ptr() + 8 * oa, b.data_ptr() + 8 * ob, lda, ldb, k, ta, tb, alpha))
        st["outs"].append(nrgb.GemmOut(st["out"].data_ptr() + 8 * o, m, m, n, 0.0, first, len(terms)))
        st["c"].append((m, n, o, first, len(terms)))
    return st


def _gemm_run(st):
    if st["slices"]:
        _context().gemm_grouped_split_dev(st["slices"], st["outs"], st["terms"], _stream())
    else:
        _context().gemm_grouped_dev(st["outs"], st["terms"], _stream())
    return st["out"]


def _gemm_exact(case, seed):
    st = _gemm_prepare(case, seed)
    for m, n, o, first, count in st["c"]:
        c = torch.zeros(m, n, device=DEV, dtype=F64)
        for a, b, k, ta, tb, oa, ob, alpha in st["keep"][first:first + count]:
            left = a[:m, oa:oa + k] if ta else a[:k, oa:oa + m].t()
            right = b[:k, ob:ob + n] if tb else b[:n, ob:ob + k].t()
            c += alpha * (left @ right)
        st["out"][o:o + m * n] = c.t().reshape(-1)
    return st["out"]


def _gemm_work(case):
    b = f = 0.0
    for m, n, terms in _gemm_shapes(case):
        b += 8.0 * m * n
        for t in terms:
            b += 8.0 * t[0] * (m + n)
            f += 2.0 * m * n * t[0]
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# allocation-free basis change
# ---------------------------------------------------------------------------
def _noalloc_sizes(case):
    s = _sizes(case["ops"] + 1, case["lo"], case["hi"], case["shape"])
    return s[:-1], s[1:]


def _noalloc_prepare(case, seed):
    nb, nk = _noalloc_sizes(case)
    g = _gen(seed)
    off, total = _layout([i * j for i, j in zip(nb, nk)])
    rand = lambda m, n: torch.randn(m, n, device=DEV, dtype=F64, generator=g) / math.sqrt(n)  # noqa: E731
    st = {"nb": nb, "nk": nk, "off": off, "out": torch.zeros(total, device=DEV, dtype=F64),
          "zb": [rand(i, i) for i in nb], "zk": [rand(j, j) for j in nk], "op": [rand(j, i) for i, j in zip(nb, nk)]}
    n = len(nb)
    ptrs = lambda ts: (ctypes.c_void_p * n)(*[t.data_ptr() for t in ts])  # noqa: E731
    st["args"] = (n, (ctypes.c_int * n)(*nb), (ctypes.c_int * n)(*nk), ptrs(st["zb"]), ptrs(st["zk"]), ptrs(st["op"]),
                  (ctypes.c_void_p * n)(*[st["out"].data_ptr() + 8 * o for o in off]))
    return st


def _noalloc_run(st):
    rc = nrgb.load().nrgb_basis_change_noalloc(*st["args"], ctypes.c_void_p(_stream()))
    if rc:
        raise RuntimeError("nrgb_basis_change_noalloc: status %d" % rc)
    return st["out"]


def _noalloc_exact(case, seed):
    st = _noalloc_prepare(case, seed)
    for zb, zk, op, o in zip(st["zb"], st["zk"], st["op"], st["off"]):
        c = zb @ op.t() @ zk.t()  # buffers are column-major: op.t() is the operator, zb its bra's Z^T
        st["out"][o:o + c.numel()] = c.t().reshape(-1)
    return st["out"]


def _noalloc_work(case):
    b = f = 0.0
    for i, j in zip(*_noalloc_sizes(case)):
        b += 8.0 * (i * i + j * j + 2 * i * j)
        f += 2.0 * i * j * (i + j)
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# one step through the step-level plan
# ---------------------------------------------------------------------------
LAMBDA, TEMPERATURE, WN, BPD, EMIN, EMAX = 2.0, 0.8, 0.3, 50, 1e-6, 1e2


def _step_shape(case):
    """Kept states of the ancestor subspaces; block b has the ancestors b .. b + 3 (cyclically)."""
    s, r = case["ancestors"], random.Random(case["shape"])
    weight = [math.exp(-((i - (s - 1) / 2) / (0.28 * s)) ** 2) * r.uniform(0.7, 1.3) for i in range(s)]
    kept = [max(1, round(case["keep"] * w / sum(weight))) for w in weight]
    return kept, [[(b + i) % s for i in range(4)] for b in range(s)]


HOPS = ((0, 1), (0, 2), (1, 3), (2, 3))


def _step_numbers(case, seed):
    """Energies, <f> blocks (first and second neighbours) and term factors, on the host."""
    kept, anc = _step_shape(case)
    r = np.random.default_rng(seed)
    s = len(kept)
    e = [np.sort(r.uniform(0.0, 5.0, k)) for k in kept]
    f = {}
    for a in range(s):
        for d in (1, 2):
            b = (a + d) % s
            f[a, b] = r.standard_normal((kept[a], kept[b])) / math.sqrt(kept[a] + kept[b])
    return kept, anc, e, f, r.uniform(0.4, 0.9, 4), r.uniform(-0.1, 0.1, 4)


def _step_prepare(case, seed):
    ctx = _context()
    kept, anc, e, f, hop, shift = _step_numbers(case, seed)
    st = {"n": len(kept), "keep": case["keep"], "kept": kept, "anc": anc}
    st["e"] = [ctx.mat_upload(x.reshape(-1, 1)) for x in e]
    st["f"] = {k: ctx.mat_upload(m) for k, m in f.items()}
    st["off"] = [np.concatenate([[0], np.cumsum([kept[a] for a in x])]).astype(int).tolist() for x in anc]
    st["dims"] = [o[4] for o in st["off"]]
    st["diag"], st["hops"], st["shift"], st["hop"] = [], [], shift, hop
    for b, x in enumerate(anc):
        o = st["off"][b]
        for i, a in enumerate(x):
            st["diag"].append(nrgb.DiagTerm(b, o[i], kept[a], st["e"][a], math.sqrt(LAMBDA), shift[i]))
        for t, (i, j) in enumerate(HOPS):
            st["hops"].append(nrgb.OffdiagTerm(b, o[i], o[j], kept[x[i]], kept[x[j]], st["f"][x[i], x[j]], hop[t]))
    st["rules"] = {"fixeps": 1e-15, "keepenergy": -1.0, "keep": case["keep"], "keepmin": 0, "safeguard": 1e-5,
                   "safeguardmax": 200, "keep_all": 0, "betabar": 1.0}
    return st


def _step_run(st):
    ctx, n, off, dims, kept_prev, anc = _context(), st["n"], st["off"], st["dims"], st["kept"], st["anc"]
    z, w, kept, egs, zsums = ctx.step(dims, st["diag"], st["hops"], st["rules"])
    energies = [ctx.mat_download(h)[:, 0] for h in w]
    # an operator between neighbouring blocks, all states of both
    outs, terms = [], []
    for b in range(n):
        c = (b + 1) % n
        outs.append(nrgb.RecalcOut(dims[b], dims[c], len(terms), 4))
        for i in range(4):
            x, y = anc[b][i], anc[c][i]
            terms.append(nrgb.RecalcTerm(z[b], off[b][i], kept_prev[x], z[c], off[c][i], kept_prev[y], st["f"][x, y],
                                         1.0 - 0.2 * i))
    op = ctx.recalc(outs, terms)
    # density matrices of the kept states, and one step back to the ancestors
    rho = [ctx.mat_upload(np.diag(np.exp(-e[:k] / TEMPERATURE)).reshape(k, k)) for e, k in zip(energies, kept)]
    outs, terms = [], []
    for s in range(n):
        outs.append(nrgb.DmOut(kept_prev[s], kept_prev[s], len(terms), 4))
        for i in range(4):
            b = (s - i) % n
            terms.append(nrgb.DmTerm(z[b], off[b][i], kept[b], z[b], off[b][i], kept[b], rho[b], 1.0 + 0.1 * i))
    back = ctx.dm_backward(outs, terms)
    rho_back = [ctx.mat_download(h) for h in back]
    # FDM spectral weights over kept and discarded states at the absolute energies
    absolute = [ctx.mat_upload(0.4 * e.reshape(-1, 1)) for e in energies]
    pairs = [nrgb.FdmPair(op[b], op[b], rho[(b + 1) % n], rho[b], absolute[(b + 1) % n], absolute[b], kept[(b + 1) % n],
                          kept[b], 1.0) for b in range(n)]
    pos, neg = ctx.spectrum_fdm(pairs, TEMPERATURE, WN, True, BPD, EMIN, EMAX)
    for h in z + w + op + rho + back + absolute:
        ctx.mat_free(h)
    return {"w": np.concatenate(energies), "kept": np.array(kept), "egs": egs, "zsums": zsums,
            "rho": np.concatenate([m.ravel() for m in rho_back]), "positive": pos, "negative": neg}


def _bin(bins, energy, weight):
    """Weights at energies onto the logarithmic grid, split linearly between the two nearest points."""
    nb = len(bins[0])
    for sign, out in ((1, bins[0]), (-1, bins[1])):
        sel = (energy < 0.0) if sign < 0 else (energy >= 0.0)
        a, w = np.abs(energy[sel]), weight[sel]
        on = np.abs(w) >= 1e-16 * a
        a, w = a[on], w[on]
        with np.errstate(divide="ignore"):
            at = np.maximum((np.log10(a) - math.floor(math.log10(EMIN))) * BPD, -1.0)
        i = np.trunc(at).astype(int)
        rem = at - i
        low, high = at <= -1.0, i >= nb - 1
        np.add.at(out, np.where(low, 0, np.minimum(i, nb - 1)), np.where(low | high, w, (1.0 - rem) * w))
        mid = ~(low | high)
        np.add.at(out, i[mid] + 1, (rem * w)[mid])


def _step_exact(case, seed):
    kept_prev, anc, e, f, hop, shift = _step_numbers(case, seed)
    n = len(kept_prev)
    ws, zs, offs = [], [], []
    for b, x in enumerate(anc):
        o = np.concatenate([[0], np.cumsum([kept_prev[a] for a in x])]).astype(int)
        h = np.diag(np.concatenate([math.sqrt(LAMBDA) * e[a] + shift[i] for i, a in enumerate(x)]))
        for t, (i, j) in enumerate(HOPS):
            m = hop[t] * f[x[i], x[j]]
            h[o[i]:o[i + 1], o[j]:o[j + 1]] += m
            h[o[j]:o[j + 1], o[i]:o[i + 1]] += m.T
        w, z = np.linalg.eigh(h)
        ws.append(w)
        zs.append(z)
        offs.append(o)
    egs = min(w[0] for w in ws)
    ws = [w - egs for w in ws]
    levels = np.sort(np.concatenate(ws))
    k = min(case["keep"], len(levels))
    most = k + 200
    while k < min(len(levels), most) and levels[k] - levels[k - 1] <= 1e-5:
        k += 1
    kept = [int(np.count_nonzero(w <= levels[k - 1])) for w in ws]
    rho = [np.exp(-w[:q] / TEMPERATURE) for w, q in zip(ws, kept)]
    back = []
    for s in range(n):
        m = 0.0
        for i in range(4):
            b = (s - i) % n
            sub = zs[b][offs[b][i]:offs[b][i + 1], :kept[b]]
            m = m + (1.0 + 0.1 * i) * ((sub * rho[b]) @ sub.T)
        back.append(m)
    nbins = int((math.ceil(math.log10(EMAX)) - math.floor(math.log10(EMIN))) * BPD + 1.0)
    bins = np.zeros(nbins), np.zeros(nbins)
    for b in range(n):
        c = (b + 1) % n
        op = 0.0
        for i in range(4):
            x, y = anc[b][i], anc[c][i]
            op = op + (1.0 - 0.2 * i) * (zs[b][offs[b][i]:offs[b][i + 1]].T @ f[x, y] @ zs[c][offs[c][i]:offs[c][i + 1]])
        ei, ej, ri, rj = 0.4 * ws[c], 0.4 * ws[b], kept[c], kept[b]
        de = ej[:, None] - ei[None, :]
        greater = op * op * WN * np.exp(-ei / TEMPERATURE)[None, :]
        greater[rj:, :ri] = op[rj:, :ri] * (op[rj:, :ri] * rho[c][None, :])
        greater[:rj, :ri] = 0.0
        lesser = op * op * WN * np.exp(-ej / TEMPERATURE)[:, None]
        lesser[:rj, ri:] = op[:rj, ri:] * (rho[b][:, None] * op[:rj, ri:])
        lesser[:rj, :ri] = 0.0
        _bin(bins, de.ravel(), greater.ravel())
        _bin(bins, de.ravel(), lesser.ravel())
    zsums = [[np.exp(-w).sum(), (w * np.exp(-w)).sum(), (w * w * np.exp(-w)).sum()] for w in ws]
    return {"w": np.concatenate(ws), "kept": None, "egs": float(egs), "zsums": np.array(zsums),
            "rho": np.concatenate([m.ravel() for m in back]), "positive": bins[0], "negative": bins[1]}


def _step_work(case):
    kept, anc = _step_shape(case)
    dims = [sum(kept[a] for a in x) for x in anc]
    w = _eig_work(dims)
    n = len(dims)
    w["bytes"] += sum(8.0 * kept[a] * (kept[(a + 1) % n] + kept[(a + 2) % n] + kept[a]) for a in range(n))
    for b in range(n):
        c = (b + 1) % n
        for i in range(4):
            x, y = kept[anc[b][i]], kept[anc[c][i]]
            w["flops"] += 2.0 * x * dims[c] * (y + dims[b])
        w["bytes"] += 16.0 * dims[b] * dims[c]
    return w


# ---------------------------------------------------------------------------
# whole runs, alone and through the run server
# ---------------------------------------------------------------------------
def _input(path, case, keep, eps_d):
    params = {"keep": keep, "specd": "A_d-A_d", "bins": 50, "savebins": True, "broaden": False,
              "prec_td": 14, "T": 1e-6 if case["nmax"] > 30 else 1e-3}
    params["dmnrg" if case.get("spectra") == "dmnrg" else "fdm"] = True
    inputgen.make_siam(path, 0.2, eps_d, 0.02, 2.0, case["nmax"], z=case["z"], params=params)


def _results(out):
    """The thermodynamics and the spectrum a run wrote, the spectrum on the whole logarithmic grid."""
    td = []
    with open(os.path.join(out, "td")) as fh:
        for line in fh:
            if not line.startswith("#") and line.strip():
                td.append([float(x) for x in line.split()])
    spectrum = np.zeros((2, 1400))
    for name in sorted(os.listdir(out)):
        if name.endswith(".bin"):
            e, w = np.fromfile(os.path.join(out, name), dtype="<f8").reshape(-1, 2).T
            spectrum[(e < 0).astype(int), np.rint((np.log10(np.abs(e)) + 24.0) * 50).astype(int)] = w
    return {"td": np.array(td), "spectrum": spectrum}


def _runs_prepare(case, seed):
    r = random.Random(seed)
    keeps = [case["keep"]] if case["kind"] == "run" else [int(k) for k in case["keeps"].split()]
    tmp = tempfile.TemporaryDirectory(prefix="nrgb_case_")
    st = {"tmp": tmp, "runs": []}
    for i, keep in enumerate(keeps):
        wd, out = os.path.join(tmp.name, "in%d" % i), os.path.join(tmp.name, "out%d" % i)
        os.makedirs(out)
        _input(wd, case, keep, -0.2 * r.random())
        st["runs"].append((wd, out))
    if case["kind"] == "served":
        _server()
    return st


def _run_run(st):
    wd, out = st["runs"][0]
    _context().run(wd, out)
    return _results(out)


def _served_run(st):
    srv = _server()
    tickets = [srv.submit(wd, out) for wd, out in st["runs"]]
    for t in tickets:
        srv.wait(t, 300.0)
    return [_results(out) for _, out in st["runs"]]


def _runs_work(case):
    """A step of Nkeep kept multiplets has about 4 Nkeep states; its blocks are
    those of the largest eight or so invariant subspaces (dimension about
    0.4 Nkeep).  Per step: the eigensolves, the recalculation of <f>, and on the
    way back the density matrix and the spectral operator."""
    f = b = 0.0
    for keep in ([case["keep"]] if case["kind"] == "run" else [int(k) for k in case["keeps"].split()]):
        n = 0.4 * keep
        f += case["nmax"] * 10 * (14.0 / 3.0 + 4.0) * n ** 3
        b += case["nmax"] * 10 * 8.0 * 4 * n ** 2
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
_KINDS = {
    "eig": (_eig_prepare, _eig_run, lambda c: _eig_work(_sizes(c["blocks"], c["lo"], c["hi"], c["shape"])), _eig_exact),
    "dsyev": (_dsyev_prepare, _dsyev_run, lambda c: _eig_work([c["n"]]), _dsyev_exact),
    "eig_recalc": (_eig_recalc_prepare, _eig_recalc_run, _eig_recalc_work, _eig_recalc_exact),
    "gemm": (_gemm_prepare, _gemm_run, _gemm_work, _gemm_exact),
    "split": (_gemm_prepare, _gemm_run, _gemm_work, _gemm_exact),
    "noalloc": (_noalloc_prepare, _noalloc_run, _noalloc_work, _noalloc_exact),
    "step": (_step_prepare, _step_run, _step_work, _step_exact),
    "run": (_runs_prepare, _run_run, _runs_work, lambda c, s: None),
    "served": (_runs_prepare, _served_run, _runs_work, lambda c, s: None),
}


def prepare(case, seed):
    st = _KINDS[case["kind"]][0](case, seed)
    st["kind"] = case["kind"]
    return st


def run(state):
    return _KINDS[state["kind"]][1](state)


def work(case):
    return _KINDS[case["kind"]][2](case)


def exact(case, seed):
    return _KINDS[case["kind"]][3](case, seed)
