"""Measured cases: what a program that contracts tensors with this package asks of it.

A case is a dict of plain values. ``op`` names the entry point:

  einsum          ``binary_einsum`` in its default (adaptive) form
  group           a ``Group`` of small contractions captured as a CUDA graph, replayed
  serve           a burst of mixed requests through a ``Server``
  permute         ``permutedims``
  unary           ``unary_einsum`` (partial sums, traces)
  hadamard        ``hadamard``
  simple_update   ``simple_update`` of one bond (contractions, SVD, truncation)

Tensors are column-major, as this package makes them, and written as
"label=extent,label=extent,...", fastest label first.
"""
import math
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PY = os.path.join(_ROOT, "muscle.jl_gb300", "python")
if _PY not in sys.path:
    sys.path.insert(0, _PY)

import muscle_gb300 as m  # noqa: E402
from muscle_gb300 import workloads as wl  # noqa: E402

DTYPES = {"float32": torch.float32, "float64": torch.float64, "complex64": torch.complex64,
          "complex128": torch.complex128}
PEPS_CAP = 1 << 22      # elements of A + B + C of a group member
SERVE_CAP = 128 << 20   # bytes of operands and output of one request
DRAW_BYTES = 2 << 30    # bytes of a drawn contraction's tensors


def listed():
    return [
        # one step of a small circuit or a test-sized network: nothing but latency
        {"name": "einsum_tiny_c64", "op": "einsum", "a": "i=4,j=3,k=6", "b": "k=6,l=5", "dtype": "complex128"},
        # two rank-4 tensors over two labels, B stored in an order a GEMM cannot take
        {"name": "einsum_rank4_c64", "op": "einsum", "a": "i=32,j=32,k=32,l=32", "b": "k=32,m=32,l=32,n=32",
         "dtype": "complex128"},
        # real tensors whose extents are multiples of nothing
        {"name": "einsum_odd_f64", "op": "einsum", "a": "i=37,j=19,k=23,l=11", "b": "l=11,m=29,k=23,n=13",
         "dtype": "float64"},
        # merging the two sites of an MPS bond at bond dimension 512, in single precision
        {"name": "einsum_bond_c32", "op": "einsum", "a": "l=512,p=4,r=512", "b": "r=512,q=4,s=512",
         "dtype": "complex64"},
        # a big real tensor reduced against an environment: long contraction, few columns, labels interleaved
        {"name": "einsum_environment_f64", "op": "einsum", "a": "a=64,b=96,c=64,d=48,e=32", "b": "e=32,c=64,f=128,a=64",
         "dtype": "float64", "out": "b,d,f"},
        # the largest contraction of the benchmark: entries over forty binades
        {"name": "einsum_large_c64", "op": "einsum", "a": "i=8192,k1=128,k2=64", "b": "k2=64,j=8192,k1=128",
         "dtype": "complex128", "values": "loguniform"},
        # neighbouring sites of a PEPS sweep, uneven bonds, one graph replayed per sweep
        {"name": "group_peps_c64", "op": "group", "members": 256, "mix": 1, "dtype": "complex128"},
        # a burst of independent requests of mixed sizes and element types
        {"name": "serve_burst", "op": "serve", "requests": 48, "mix": 5},
        # the permutation in front of a library GEMM
        {"name": "permute_rank5_f64", "op": "permute", "x": "a=64,b=96,c=64,d=48,e=32", "out": "b,d,a,c,e",
         "dtype": "float64"},
        # summing a middle label out of a large tensor
        {"name": "unary_sum_c64", "op": "unary", "x": "a=4096,b=1024,c=32", "out": "a,c", "dtype": "complex128"},
        # weighting a tensor's bond by its singular values
        {"name": "hadamard_c64", "op": "hadamard", "a": "l=96,p=2,r=1531", "b": "r=1531", "dtype": "complex128"},
        # a two-site gate on one bond, truncated back to the bond dimension
        {"name": "simple_update_c64", "op": "simple_update", "chi": 32, "phys": 2, "dtype": "complex128"},
    ]


# --------------------------------------------------------------------------- drawing
def _split(rng, total, parts):
    """`parts` extents whose product is about `total`."""
    if parts == 0:
        return []
    w = [rng.random() + 0.25 for _ in range(parts)]
    return [max(1, round(total ** (x / sum(w)))) for x in w]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _text(labels, ext):
    return ",".join("%s=%d" % (i, ext[i]) for i in labels)


def _draw_einsum(rng):
    while True:
        dtype = rng.choice(["complex128", "complex128", "float64", "float64", "complex64", "float32"])
        cx = dtype.startswith("complex")
        mnk = _log(rng, 1e4, 1.5e12) / (8.0 if cx else 2.0)
        share = [rng.random() + 0.4 for _ in range(3)]
        em, en, ek = (_split(rng, mnk ** (s / sum(share)), rng.randint(1, 3)) for s in share)
        eb = [rng.randint(2, 6)] if rng.random() < 0.15 else []
        names = ["x%d" % i for i in range(len(em) + len(en) + len(ek) + len(eb))]
        ext = dict(zip(names, em + en + ek + eb))
        lm, ln = names[:len(em)], names[len(em):len(em) + len(en)]
        lk, lb = names[len(em) + len(en):len(names) - len(eb)], names[len(names) - len(eb):]
        ia, ib, ic = lm + lk + lb, lk + ln + lb, lm + ln + lb
        for labels in (ia, ib, ic):
            rng.shuffle(labels)
        nbytes = 16 * sum(math.prod(ext[i] for i in labels) for labels in (ia, ib, ic))
        if nbytes > DRAW_BYTES:
            continue
        c = {"op": "einsum", "a": _text(ia, ext), "b": _text(ib, ext), "out": ",".join(ic), "dtype": dtype}
        if cx and rng.random() < 0.15:
            c["dtype_b"] = "float64" if dtype == "complex128" else "float32"
        if dtype in ("complex128", "float64") and rng.random() < 0.25:
            c["values"] = "loguniform"
        return c


def _draw_shape(rng, lo, hi, ranks):
    labels = ["a", "b", "c", "d", "e"][:rng.randint(*ranks)]
    return labels, dict(zip(labels, _split(rng, _log(rng, lo, hi), len(labels))))


def draw(rng):
    op = rng.choice(["einsum"] * 6 + ["group", "serve", "permute", "unary", "hadamard", "simple_update"])
    dtype = rng.choice(["complex128", "float64", "complex64", "float32"])
    if op == "einsum":
        return _draw_einsum(rng)
    if op == "group":
        return {"op": op, "members": round(_log(rng, 16, 384)), "mix": rng.randint(100, 10**6),
                "dtype": rng.choice(["complex128", "complex64"])}
    if op == "serve":
        return {"op": op, "requests": rng.randint(6, 60), "mix": rng.randint(100, 10**6)}
    if op == "simple_update":
        phys = rng.randint(2, 3)
        return {"op": op, "chi": round(_log(rng, 6, 96 / phys)), "phys": phys, "dtype": rng.choice(["complex128", "float64"])}
    if op == "permute":
        labels, ext = _draw_shape(rng, 1e4, 2.5e8, (2, 5))
        out = labels[:]
        while out == labels:
            rng.shuffle(out)
        return {"op": op, "x": _text(labels, ext), "out": ",".join(out), "dtype": dtype}
    labels, ext = _draw_shape(rng, 1e4, 2.0e8, (2, 4))
    if op == "hadamard":
        keep = rng.sample(labels, rng.randint(1, len(labels)))
        return {"op": op, "a": _text(labels, ext), "b": _text(keep, ext), "dtype": dtype}
    if rng.random() < 0.25:  # a trace over the outer pair of labels
        n = round(_log(rng, 16, 2000))
        return {"op": op, "x": "t=%d,a=%d,t=%d" % (n, round(_log(rng, 1, 48)), n), "out": "a", "dtype": dtype}
    kept = rng.sample(labels, rng.randint(0, len(labels) - 1))
    keep = [i for i in labels if i in kept]
    return {"op": op, "x": _text(labels, ext), "out": ",".join(keep), "dtype": dtype}


# --------------------------------------------------------------------------- shapes
def _spec(text):
    parts = [p.split("=") for p in text.split(",")]
    return [p[0] for p in parts], [int(p[1]) for p in parts]


def _names(text):
    return [i for i in text.split(",") if i]


def _einsum_spec(case):
    (ia, sa), (ib, sb) = _spec(case["a"]), _spec(case["b"])
    ext = dict(zip(ia + ib, sa + sb))
    ic = _names(case["out"]) if "out" in case else [i for i in ia if i not in ib] + [i for i in ib if i not in ia]
    return ia, sa, ib, sb, ic, [ext[i] for i in ic]


def _group_specs(case):
    """Members as (ia, ea, ib, eb, ic, ec): a rank-5 site (physical extent 2,
    four bonds of one dimension) and a neighbour over one to three bonds."""
    rng = random.Random(case["mix"])
    out = []
    while len(out) < case["members"]:
        chi, nsh = rng.choice(wl.PEPS_CHI), rng.randint(1, 3)
        if 4 * chi ** 4 + 4 * chi ** (2 * (4 - nsh)) > PEPS_CAP:
            continue
        bonds = ["u", "r", "d", "l"]
        shared = rng.sample(bonds, nsh)
        free = ["x%d" % t for t in range(4 - nsh)]
        ia, ib = ["p"] + bonds, ["q"] + shared + free
        ic = ["p"] + [i for i in bonds if i not in shared] + ["q"] + free
        out.append((ia, [2] + [chi] * 4, ib, [2] + [chi] * 4, ic,
                    [2] + [chi] * (4 - nsh) + [2] + [chi] * (4 - nsh)))
    return out


def _serve_specs(case):
    """Requests as (shape_a, ia, shape_b, ib, ic, shape_c, dtype)."""
    rng = np.random.default_rng(case["mix"])
    kinds = {np.complex128: torch.complex128, np.float64: torch.float64, np.complex64: torch.complex64}
    out = []
    while len(out) < case["requests"]:
        sa, ia, sb, ib, ic, dt, _ = wl.serve_request(rng)
        ext = dict(zip(ia + ib, sa + sb))
        sc = [ext[i] for i in ic]
        if (math.prod(sa) + math.prod(sb) + math.prod(sc)) * np.dtype(dt).itemsize <= SERVE_CAP:
            out.append(([int(x) for x in sa], [str(i) for i in ia], [int(x) for x in sb], [str(i) for i in ib],
                        [str(i) for i in ic], [int(x) for x in sc], kinds[dt]))
    return out


def _update_spec(case):
    chi, d = case["chi"], case["phys"]
    return (["p1", "l", "b"], [d, chi, chi]), (["p2", "b", "r"], [d, chi, chi]), (["p1", "p2", "q1", "q2"], [d] * 4)


# --------------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _fill(gen, shape, dtype, values="normal", scale=1.0):
    """A column-major array of standard normal entries, or of magnitudes
    2^U(-20, 20) with a uniform phase (a random sign when real)."""
    rev = list(reversed(shape))
    if values == "loguniform":
        x = torch.exp2(torch.rand(rev, dtype=torch.float64, device="cuda", generator=gen) * 40 - 20)
        u = torch.rand(rev, dtype=torch.float64, device="cuda", generator=gen)
        x = torch.polar(x, u * (2 * math.pi)) if dtype.is_complex else torch.where(u < 0.5, -x, x)
        x = x.to(dtype)
    else:
        x = torch.randn(rev, dtype=dtype, device="cuda", generator=gen)
        if scale != 1.0:
            x *= scale
    return x.permute(*reversed(range(len(rev)))) if rev else x


def _einsum_inputs(case, seed):
    ia, sa, ib, sb, ic, _ = _einsum_spec(case)
    g, values = _gen(seed), case.get("values", "normal")
    a = _fill(g, sa, DTYPES[case["dtype"]], values)
    b = _fill(g, sb, DTYPES[case.get("dtype_b", case["dtype"])], values)
    return (a, ia), (b, ib), ic


def _group_inputs(case, seed):
    g, dt = _gen(seed), DTYPES[case["dtype"]]
    out = []
    for ia, ea, ib, eb, ic, ec in _group_specs(case):
        s = ea[1] ** -0.5
        out.append(((_fill(g, ea, dt, scale=s), ia), (_fill(g, eb, dt, scale=s), ib), ic, ec))
    return out


def _serve_inputs(case, seed):
    g = _gen(seed)
    return [((_fill(g, sa, dt), ia), (_fill(g, sb, dt), ib), ic) for sa, ia, sb, ib, ic, _, dt in _serve_specs(case)]


def _one_input(case, seed, key):
    labels, shape = _spec(case[key])
    return _fill(_gen(seed), shape, DTYPES[case["dtype"]]), labels


def _hadamard_inputs(case, seed):
    g, dt = _gen(seed), DTYPES[case["dtype"]]
    (ia, sa), (ib, sb) = _spec(case["a"]), _spec(case["b"])
    return (_fill(g, sa, dt), ia), (_fill(g, sb, dt), ib)


def _update_inputs(case, seed):
    g, dt = _gen(seed), DTYPES[case["dtype"]]
    return [(_fill(g, s, dt), i) for i, s in _update_spec(case)]


def prepare(case, seed):
    op = case["op"]
    if op == "einsum":
        (a, ia), (b, ib), ic = _einsum_inputs(case, seed)
        return {"op": op, "a": m.Tensor(a, ia), "b": m.Tensor(b, ib), "out": ic}
    if op == "group":
        members = _group_inputs(case, seed)
        classes = {}
        for k, (_, _, ic, ec) in enumerate(members):
            classes.setdefault(tuple(ec), []).append(k)
        outs, items = [], [None] * len(members)
        for ec, ks in sorted(classes.items()):  # the outputs of one shape lie together
            buf = torch.empty([len(ks)] + list(reversed(ec)), dtype=DTYPES[case["dtype"]], device="cuda")
            outs.append(buf)
            for j, k in enumerate(ks):
                (a, ia), (b, ib), ic, _ = members[k]
                c = buf[j].permute(*reversed(range(len(ec))))
                items[k] = (m.Tensor(c, ic), m.Tensor(a, ia), m.Tensor(b, ib))
        group = m.Group(items)
        return {"op": op, "group": group, "graph": group.capture(), "outs": outs}
    if op == "serve":
        return {"op": op, "server": m.Server(),
                "requests": [(m.Tensor(a, ia), m.Tensor(b, ib), ic) for (a, ia), (b, ib), ic in _serve_inputs(case, seed)]}
    if op == "hadamard":
        (a, ia), (b, ib) = _hadamard_inputs(case, seed)
        return {"op": op, "a": m.Tensor(a, ia), "b": m.Tensor(b, ib)}
    if op == "simple_update":
        A, B, G = (m.Tensor(x, i) for x, i in _update_inputs(case, seed))
        return {"op": op, "a": A, "b": B, "g": G, "maxdim": case["chi"]}
    x, ix = _one_input(case, seed, "x")
    return {"op": op, "x": m.Tensor(x, ix), "out": _names(case["out"])}


def run(state):
    op = state["op"]
    if op == "einsum":
        return m.binary_einsum(state["a"], state["b"], out=state["out"]).data
    if op == "group":
        state["graph"].replay()
        return state["outs"]
    if op == "serve":
        pending = [state["server"].submit(a, b, out=ic) for a, b, ic in state["requests"]]
        return [p.result().data for p in pending]
    if op == "permute":
        return m.permutedims(state["x"], state["out"]).data
    if op == "unary":
        return m.unary_einsum(state["x"], out=state["out"]).data
    if op == "hadamard":
        return m.hadamard(state["a"], state["b"]).data
    u, s, v = m.simple_update(state["a"], "p1", state["b"], "p2", "b", state["g"], "q1", "q2", normalize=True,
                              maxdim=state["maxdim"])
    return [u.data, s.data, v.data]


# --------------------------------------------------------------------------- what a pass cannot do without
def _size(dtype):
    return torch.empty((), dtype=dtype).element_size()


def _pair_work(sa, sb, sc, ka, kb):
    kc = torch.promote_types(ka, kb)
    na, nb, nc = math.prod(sa), math.prod(sb), math.prod(sc)
    return na * _size(ka) + nb * _size(kb) + nc * _size(kc), kc.is_complex


def work(case):
    op = case["op"]
    if op == "einsum":
        ia, sa, ib, sb, ic, sc = _einsum_spec(case)
        ka = DTYPES[case["dtype"]]
        nbytes, cx = _pair_work(sa, sb, sc, ka, DTYPES[case.get("dtype_b", case["dtype"])])
        return {"bytes": nbytes, "flops": (8.0 if cx else 2.0) * math.prod(dict(zip(ia + ib, sa + sb)).values())}
    if op in ("group", "serve"):
        nbytes, flops = 0, 0.0
        if op == "group":
            specs = [(ea, ia, eb, ib, ec, DTYPES[case["dtype"]]) for ia, ea, ib, eb, ic, ec in _group_specs(case)]
        else:
            specs = [(sa, ia, sb, ib, sc, dt) for sa, ia, sb, ib, ic, sc, dt in _serve_specs(case)]
        for sa, ia, sb, ib, sc, dt in specs:
            b, cx = _pair_work(sa, sb, sc, dt, dt)
            nbytes += b
            flops += (8.0 if cx else 2.0) * math.prod(dict(zip(ia + ib, sa + sb)).values())
        return {"bytes": nbytes, "flops": flops}
    dt = DTYPES[case["dtype"]]
    es, cx = _size(dt), dt.is_complex
    if op == "permute":
        return {"bytes": 2 * es * math.prod(_spec(case["x"])[1]), "flops": 0.0}
    if op == "unary":
        ix, sx = _spec(case["x"])
        ext = dict(zip(ix, sx))
        read, written = math.prod(ext.values()), math.prod(ext[i] for i in _names(case["out"]))
        return {"bytes": es * (read + written), "flops": (2.0 if cx else 1.0) * read}
    if op == "hadamard":
        na, nb = math.prod(_spec(case["a"])[1]), math.prod(_spec(case["b"])[1])
        return {"bytes": es * (2 * na + nb), "flops": (6.0 if cx else 1.0) * na}
    # the two contractions, and a dense factorisation of the n x n matrix at
    # the cost of a bidiagonalisation with both factors
    chi, d = case["chi"], case["phys"]
    n, f = chi * d, 8.0 if cx else 2.0
    flops = f * (d * d * chi ** 3 + d ** 4 * chi * chi) + (4.0 if cx else 1.0) * 12.0 * n ** 3
    return {"bytes": es * (2 * d * chi * chi + d ** 4 + 2 * n * chi) + 8 * chi, "flops": flops}


# --------------------------------------------------------------------------- in 64 bits, without this package
def _wide(x):
    return x.to(torch.complex128 if x.is_complex() else torch.float64)


def _ein(tensors, out):
    """torch.einsum over named labels, in 64 bits."""
    xs = [_wide(x) for x, _ in tensors]
    kind = torch.complex128 if any(x.is_complex() for x in xs) else torch.float64
    ids = {}
    args = []
    for x, (_, labels) in zip(xs, tensors):
        args += [x.to(kind), [ids.setdefault(i, len(ids)) for i in labels]]
    return torch.einsum(*args, [ids[i] for i in out])


def exact(case, seed):
    op = case["op"]
    if op == "einsum":
        a, b, ic = _einsum_inputs(case, seed)
        return _ein([a, b], ic)
    if op == "group":
        classes = {}
        for a, b, ic, ec in _group_inputs(case, seed):
            c = _ein([a, b], ic)
            classes.setdefault(tuple(ec), []).append(c.permute(*reversed(range(c.dim()))).contiguous())
        return [torch.stack(v) for _, v in sorted(classes.items())]
    if op == "serve":
        return [_ein([a, b], ic) for a, b, ic in _serve_inputs(case, seed)]
    if op == "permute":
        x, ix = _one_input(case, seed, "x")
        return x.permute(*[ix.index(i) for i in _names(case["out"])])
    if op == "unary":
        x, ix = _one_input(case, seed, "x")
        return _ein([(x, ix)], _names(case["out"]))
    if op == "hadamard":
        (a, ia), (b, ib) = _hadamard_inputs(case, seed)
        return _ein([(a, ia), (b, ib)], ia)
    a, b, g = _update_inputs(case, seed)
    theta = _ein([a, b, g], ["q1", "l", "q2", "r"])
    n = case["phys"] * case["chi"]
    s = torch.linalg.svdvals(theta.reshape(n, n).cpu())[:case["chi"]]
    return [None, s / torch.linalg.vector_norm(s), None]  # singular vectors are unique up to a phase
