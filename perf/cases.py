"""The measured workloads: what an iterative many-body (coupled-cluster) program
does with this library, through its Python entry points, on tensors that stay on
the GPU.

A case is a dict of plain values; `prepare` makes its inputs from a seed, `run`
makes one pass, `exact` gives the same outputs from torch in 64 bits. Labels
a-f are virtual (extent v), i-n occupied (extent o) unless a case says
otherwise. Tensors are stored with the first label of the storage order fastest,
as TBLIS's column-major varrays are.
"""
import itertools
import math
import random

import torch

import tblis_b200 as tb

DTYPES = {"f32": torch.float32, "f64": torch.float64, "c64": torch.complex64, "c128": torch.complex128}

# contraction terms: labels of A, B, C, their storage orders (first = fastest)
# and whether C is accumulated into (a residual that starts as a copy of its
# driver term) or overwritten
TERMS = {
    # particle-particle ladder, the most expensive term of coupled cluster
    "ladder": {"A": "abef", "B": "efij", "C": "abij", "sA": "abef", "sB": "efij", "sC": "abij", "add": False},
    # ring term: every group interleaves in storage, so no operand is a plain
    # matrix, and the result is added to a residual
    "ring": {"A": "aeim", "B": "mbej", "C": "aibj", "sA": "aeim", "sB": "mbej", "sC": "aibj", "add": True},
    # the same with operands stored in other orders (permuted amplitudes)
    "ring2": {"A": "aeim", "B": "mbej", "C": "aibj", "sA": "imae", "sB": "ejbm", "sC": "abij", "add": True},
    # one-particle intermediate: a small result, a long contraction
    "fock": {"A": "mnaf", "B": "mnef", "C": "ae", "sA": "afmn", "sB": "efmn", "sC": "ae", "add": False},
}

# orbitals per irrep of a D2h molecule (8 irreps), and of a C2v one (4)
GROUPS = {
    8: ([12, 4, 8, 6, 10, 3, 7, 5], [60, 22, 40, 30, 52, 14, 36, 26]),
    4: ([9, 3, 5, 4], [41, 17, 29, 20]),
}


def listed():
    return [
        # one term of a small molecule or of a fragment: latency and launches count
        {"name": "mult_small", "kind": "mult", "term": "ladder", "o": 4, "v": 8, "dtype": "f64"},
        # the plain dense contraction with every extent 24
        {"name": "mult_24", "kind": "mult", "term": "ladder", "o": 24, "v": 24, "dtype": "f64"},
        # a large ring term in double precision, the bulk of a CCSD iteration beside the ladder
        {"name": "ring_f64", "kind": "mult", "term": "ring", "o": 48, "v": 160, "dtype": "f64"},
        # an intermediate with a small result and a long sum, odd extents
        {"name": "fock_f64", "kind": "mult", "term": "fock", "o": 31, "v": 97, "dtype": "f64"},
        # the ladder with a requested normwise error of 1e-12, wide exponent range
        {"name": "ladder_tol", "kind": "mult", "term": "ladder", "o": 48, "v": 160, "dtype": "f64",
         "config": "b200_ozaki_i8", "spread": 20},
        # the ladder in single precision (a low-accuracy start of an iteration), odd extents
        {"name": "ladder_f32", "kind": "mult", "term": "ladder", "o": 37, "v": 101, "dtype": "f32"},
        # a ring term with complex orbitals (relativistic, periodic), permuted storage
        {"name": "ring_c128", "kind": "mult", "term": "ring2", "o": 24, "v": 72, "dtype": "c128"},
        # many small independent contractions (local correlation domains) in one call
        {"name": "batch", "kind": "batch", "count": 2000, "lo": 4, "hi": 32},
        # the ladder of a symmetric molecule, block sparse
        {"name": "dpd_ladder", "kind": "dpd_mult", "nirrep": 8, "scale": 1.0},
        # a transpose of the amplitudes
        {"name": "transpose", "kind": "transpose", "o": 48, "v": 160, "dtype": "f64", "to": "ijab"},
        # the end of an iteration: symmetrise the residual, its norm, the energy; odd extents
        {"name": "update", "kind": "update", "o": 31, "v": 97, "dtype": "f64"},
        # the same on block-sparse amplitudes
        {"name": "dpd_update", "kind": "dpd_update", "nirrep": 8, "scale": 1.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mult", "mult", "mult", "mult", "tol", "batch", "dpd_mult", "transpose", "update", "dpd_update"])
    while True:
        if kind == "mult":
            c = {"kind": "mult", "term": rng.choice(sorted(TERMS)), "o": _log(rng, 4, 48), "v": _log(rng, 8, 160),
                 "dtype": rng.choice(["f64", "f64", "f64", "f32", "c64", "c128"])}
            limit = 0.9e12
        elif kind == "tol":
            c = {"kind": "mult", "term": rng.choice(["ladder", "ring"]), "o": _log(rng, 16, 48),
                 "v": _log(rng, 64, 160), "dtype": "f64", "config": "b200_ozaki_i8", "spread": rng.choice([0, 8, 20])}
            limit = 3.1e12
        elif kind == "batch":
            lo = rng.randint(3, 12)
            c = {"kind": "batch", "count": _log(rng, 50, 2000), "lo": lo, "hi": rng.randint(lo + 2, 32)}
            limit = 0.2e12
        elif kind in ("dpd_mult", "dpd_update"):
            c = {"kind": kind, "nirrep": rng.choice([4, 8]), "scale": round(rng.uniform(0.25, 1.0), 3)}
            limit = 0.9e12
        else:
            c = {"kind": kind, "o": _log(rng, 4, 48), "v": _log(rng, 8, 160),
                 "dtype": rng.choice(["f64", "f64", "c128"])}
            if kind == "transpose":
                c["dtype"] = rng.choice(["f64", "f64", "f32", "c64", "c128"])
                c["to"] = "".join(rng.sample("abij", 4))
            limit = 0.9e12
        w = work(c)
        if w["flops"] <= limit and w["bytes"] <= 6e9:
            return c


# ---- inputs ---------------------------------------------------------------------------


def _ext(case, labels):
    return [case["v"] if c in "abcdef" else case["o"] for c in labels]


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _stored(case, labels, order, g=None):
    """A tensor with the given labels, stored with order[0] fastest; uniform
    in (-1, 1) (times 2^k, k in [-spread, spread], when the case has a
    spread), or uninitialised without a generator."""
    rev = order[::-1]
    dt = DTYPES[case["dtype"]]
    t = torch.empty(_ext(case, rev), dtype=dt, device="cuda")
    if g is not None:
        r = torch.view_as_real(t) if dt.is_complex else t
        r.uniform_(-1.0, 1.0, generator=g)
        s = case.get("spread", 0)
        if s:
            r.mul_(torch.exp2(torch.randint(-s, s + 1, r.shape, generator=g, device="cuda", dtype=torch.int32).to(r.dtype)))
    return t.permute([rev.index(c) for c in labels])


def _mult_inputs(case, seed):
    t = TERMS[case["term"]]
    g = _gen(seed)
    A = _stored(case, t["A"], t["sA"], g)
    B = _stored(case, t["B"], t["sB"], g)
    D = _stored(case, t["C"], t["sC"], g) if t["add"] else None     # the driver term
    return t, A, B, D


def _batch_inputs(case, seed):
    rnd = random.Random(1000 * case["count"] + 32 * case["lo"] + case["hi"])
    g = _gen(seed)
    out = []
    for _ in range(case["count"]):
        l = {c: rnd.randint(case["lo"], case["hi"]) for c in "abefij"}
        ia, ib, ic = ("".join(rnd.sample(s, 4)) for s in ("abef", "efij", "abij"))
        out.append((l, ia, ib, ic))
    # one allocation per operand kind, as a program with an arena would keep them
    sizes = [[math.prod(l[c] for c in ix) for l, *_ in out] for ix in ("abef", "efij")]
    flat = [torch.empty(sum(s), dtype=torch.float64, device="cuda").uniform_(-1.0, 1.0, generator=g) for s in sizes]
    parts = [f.split(s) for f, s in zip(flat, sizes)]
    items = []
    for n, (l, ia, ib, ic) in enumerate(out):
        items.append((parts[0][n].view([l[c] for c in ia]), ia, parts[1][n].view([l[c] for c in ib]), ib,
                      [l[c] for c in ic], ic))
    return items


# ---- block-sparse tensors ---------------------------------------------------------------


def _irreps(case):
    occ, vir = GROUPS[case["nirrep"]]
    s = case["scale"]
    return [max(1, round(x * s)) for x in occ], [max(1, round(x * s)) for x in vir]


def _flat(lens, g):
    """Storage of a totally symmetric block-sparse tensor, uniform in (-1, 1)."""
    return torch.empty(_sym(lens), dtype=torch.float64, device="cuda").uniform_(-1.0, 1.0, generator=g)


def _dpd(lens, data=None):
    data = torch.empty(_sym(lens), dtype=torch.float64, device="cuda") if data is None else data
    return tb.DpdTensor(0, len(lens[0]), lens, data)


def _dpd_update_inputs(o, v, seed):
    """Block-sparse amplitudes X[abij] and integrals V[ijab] = X + noise."""
    g = _gen(seed)
    lx, lv = [v, v, o, o], [o, o, v, v]
    x, w = _flat(lx, g), _flat(lv, g).mul_(0.5)
    bv = _blocks(lv)
    for (a, b, i, j), blk in _blocks(lx).items():
        _view(w, bv[i, j, a, b]).add_(_view(x, blk).permute(2, 3, 0, 1))
    return x, w


def _update_inputs(case, seed):
    """Amplitudes and integrals in the transposed order. Amplitudes follow the
    integrals (they are the integrals over energy differences to first order),
    so the energy is a sum of mostly one sign."""
    g = _gen(seed)
    X, V = _stored(case, "abij", "abij", g), _stored(case, "ijab", "ijab", g)
    V.mul_(0.5).add_(X.permute(2, 3, 0, 1).conj())
    return X, V


def prepare(case, seed):
    s = {"case": case}
    kind = case["kind"]
    if kind == "mult":
        t, s["A"], s["B"], s["D"] = _mult_inputs(case, seed)
        s["C"] = _stored(case, t["C"], t["sC"])
        s["cfg"] = tb.get_config(case["config"]) if case.get("config") else None
    elif kind == "batch":
        inputs = _batch_inputs(case, seed)
        sizes = [math.prod(shape) for *_, shape, _ in inputs]
        s["C"] = torch.empty(sum(sizes), dtype=torch.float64, device="cuda")
        s["batch"] = tb.PreparedBatch([(1.0, a, ia, b, ib, 0.0, c.view(shape), ic)
                                       for (a, ia, b, ib, shape, ic), c in zip(inputs, s["C"].split(sizes))])
    elif kind == "dpd_mult":
        o, v = _irreps(case)
        g = _gen(seed)
        s["A"], s["B"] = _dpd([v] * 4, _flat([v] * 4, g)), _dpd([v, v, o, o], _flat([v, v, o, o], g))
        s["C"] = _dpd([v, v, o, o])
    elif kind == "dpd_update":
        o, v = _irreps(case)
        x, w = _dpd_update_inputs(o, v, seed)
        s["X"], s["V"], s["R"] = _dpd([v, v, o, o], x), _dpd([o, o, v, v], w), _dpd([v, v, o, o])
    elif kind == "transpose":
        s["C"] = _stored(case, "abij", "abij", _gen(seed))
        s["D"] = _stored(case, case["to"], case["to"])
    else:
        s["X"], s["V"] = _update_inputs(case, seed)
        s["R"] = _stored(case, "abij", "abij")
    return s


def _parts(z):
    return [z.real, z.imag] if isinstance(z, complex) else z


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "mult":
        t = TERMS[case["term"]]
        if t["add"]:
            tb.add(1.0, s["D"], t["C"], 0.0, s["C"], t["C"])
        tb.mult(1.0, s["A"], t["A"], s["B"], t["B"], 1.0 if t["add"] else 0.0, s["C"], t["C"], cfg=s["cfg"])
        return s["C"]
    if kind == "batch":
        s["batch"].run()
        return s["C"]
    if kind == "dpd_mult":
        tb.dpd_mult(1.0, s["A"], "abef", s["B"], "efij", 0.0, s["C"], "abij")
        return s["C"].data
    if kind == "dpd_update":
        tb.dpd_add(1.0, s["X"], "abij", 0.0, s["R"], "abij")
        tb.dpd_add(1.0, s["X"], "baji", 1.0, s["R"], "abij")
        norm, _ = tb.dpd_reduce(tb.REDUCE_NORM_2, s["R"], "abij")
        return s["R"].data, norm, tb.dpd_dot(s["R"], "abij", s["V"], "ijab")
    if kind == "transpose":
        tb.add(1.0, s["C"], "abij", 0.0, s["D"], case["to"])
        return s["D"]
    tb.add(1.0, s["X"], "abij", 0.0, s["R"], "abij")
    tb.add(1.0, s["X"], "baji", 1.0, s["R"], "abij")
    norm, _ = tb.reduce(tb.REDUCE_NORM_2, s["R"], "abij")
    return s["R"], _parts(norm), _parts(tb.dot(s["R"], "abij", s["V"], "ijab"))


# ---- what a pass cannot do without -----------------------------------------------------


def _sym(dims):
    """Elements of a totally symmetric block-sparse tensor."""
    n = len(dims[0])
    c = [1 if h == 0 else 0 for h in range(n)]
    for d in dims:
        c = [sum(c[h ^ x] * d[x] for x in range(n)) for h in range(n)]
    return c[0]


def work(case):
    kind = case["kind"]
    if kind == "mult":
        t = TERMS[case["term"]]
        es = DTYPES[case["dtype"]].itemsize
        n = [math.prod(_ext(case, t[x])) for x in "ABC"]
        mnk = math.prod(_ext(case, sorted(set(t["A"] + t["B"]))))
        return {"bytes": es * (n[0] + n[1] + n[2] * (2 if t["add"] else 1)),
                "flops": (8.0 if case["dtype"][0] == "c" else 2.0) * mnk}
    if kind == "batch":
        rnd = random.Random(1000 * case["count"] + 32 * case["lo"] + case["hi"])
        by = fl = 0
        for _ in range(case["count"]):
            l = {c: rnd.randint(case["lo"], case["hi"]) for c in "abefij"}
            for s in ("abef", "efij", "abij"):
                rnd.sample(s, 4)
                by += 8 * math.prod(l[c] for c in s)
            fl += 2.0 * math.prod(l.values())
        return {"bytes": by, "flops": fl}
    if kind in ("dpd_mult", "dpd_update"):
        o, v = _irreps(case)
        t2 = _sym([v, v, o, o])
        if kind == "dpd_update":
            return {"bytes": 8 * 3 * t2, "flops": 5.0 * t2}
        n = case["nirrep"]
        pair = lambda x, h: sum(x[g] * x[g ^ h] for g in range(n))
        return {"bytes": 8 * (_sym([v] * 4) + 2 * t2), "flops": sum(2.0 * pair(v, h) ** 2 * pair(o, h) for h in range(n))}
    es = DTYPES[case["dtype"]].itemsize
    n = (case["o"] * case["v"]) ** 2
    return {"bytes": es * n * (2 if kind == "transpose" else 3), "flops": 0.0 if kind == "transpose" else 5.0 * n}


# ---- the same outputs in 64 bits --------------------------------------------------------


def _wide(t):
    return t.to(torch.complex128 if t.dtype.is_complex else torch.float64)


def _einsum(labels, A, B):
    return torch.einsum(labels, _wide(A), _wide(B))


def _blocks(lens):
    """Views of the blocks of a totally symmetric tensor in its storage (the
    last label fastest, its irreps nested inside those of the labels before
    it): {irreps: (offset, lengths, strides)}."""
    nd, n = len(lens), len(lens[0])
    # size[d][h]: elements of the labels d.. with irrep product h
    size = [None] * nd + [[1 if h == 0 else 0 for h in range(n)]]
    for d in reversed(range(nd)):
        size[d] = [sum(size[d + 1][h ^ x] * lens[d][x] for x in range(n)) for h in range(n)]
    out = {}
    for irr in itertools.product(range(n), repeat=nd - 1):
        last = 0
        for x in irr:
            last ^= x
        irr = irr + (last,)
        off, strides, h = 0, [0] * nd, 0
        for d in reversed(range(nd)):
            strides[d] = size[d + 1][h]
            h ^= irr[d]
            off += sum(size[d + 1][x ^ h] * lens[d][x] for x in range(irr[d]))
        out[irr] = (off, [lens[d][irr[d]] for d in range(nd)], strides)
    return out


def _view(data, block):
    off, shape, strides = block
    return torch.as_strided(data, shape, strides, off)


def exact(case, seed):
    kind = case["kind"]
    if kind == "mult":
        t, A, B, D = _mult_inputs(case, seed)
        out = _einsum("%s,%s->%s" % (t["A"], t["B"], t["C"]), A, B)
        return out + _wide(D) if t["add"] else out
    if kind == "batch":
        return torch.cat([_einsum("%s,%s->%s" % (ia, ib, ic), a, b).reshape(-1)
                          for a, ia, b, ib, _, ic in _batch_inputs(case, seed)])
    if kind == "dpd_mult":
        o, v = _irreps(case)
        g = _gen(seed)
        la, lb = [v] * 4, [v, v, o, o]
        a, b = _flat(la, g), _flat(lb, g)
        c = torch.zeros(_sym(lb), dtype=torch.float64, device="cuda")
        ba, bb = _blocks(la), _blocks(lb)
        for irr, blk in bb.items():
            x = _view(c, blk)
            for e in range(case["nirrep"]):
                f = e ^ irr[0] ^ irr[1]
                x += torch.einsum("abef,efij->abij", _view(a, ba[irr[0], irr[1], e, f]), _view(b, bb[e, f, irr[2], irr[3]]))
        return c
    if kind == "dpd_update":
        o, v = _irreps(case)
        x, w = _dpd_update_inputs(o, v, seed)
        r = torch.empty_like(x)
        bx, bv = _blocks([v, v, o, o]), _blocks([o, o, v, v])
        dot = 0.0
        for (a, b, i, j), blk in bx.items():
            y = _view(r, blk)
            y.copy_(_view(x, blk) + _view(x, bx[b, a, j, i]).permute(1, 0, 3, 2))
            dot += (y * _view(w, bv[i, j, a, b]).permute(2, 3, 0, 1)).sum().item()
        return r, torch.linalg.vector_norm(r).item(), dot
    if kind == "transpose":
        C = _wide(_stored(case, "abij", "abij", _gen(seed)))
        return C.permute(["abij".index(c) for c in case["to"]])
    X, V = (_wide(x) for x in _update_inputs(case, seed))
    R = X + X.permute(1, 0, 3, 2)
    # the norm of a complex tensor comes back as a complex number
    norm = torch.linalg.vector_norm(R).to(R.dtype).item()
    return R, _parts(norm), _parts((R * V.permute(2, 3, 0, 1)).sum().item())
