"""The workloads whose time is measured: what programs have this library do.

Every case is one or a few calls of the Python host API (t1m_gb300, the mirror
of the C-ABI and of the C++ header) on buffers the caller owns.  Sizes are
those of the repository's configurations, tests and benchmark (the reference's
example contraction, the 48^4 and permuted drop-in contractions, the 4096^3
product, the tensor-network sweep, the adjoint and the ring chain) and ragged
sizes near them.

A case is a dict of plain values; ``kind`` selects the entry point:

* ``contract``: one contraction, device or pinned host buffers;
* ``vjp``: the adjoint of one contraction (both gradients);
* ``sweep``: a grouped batch of sweep updates, planned once, launched per pass;
* ``ring``: the gradients of a ring of four tensors (ContractionChain).
"""
import math
import random

import torch

import t1m_gb300 as t1m
from t1m_gb300.chain import ContractionChain

_TORCH = {"complex64": torch.complex64, "complex128": torch.complex128,
          "float32": torch.float32, "float64": torch.float64}
_BYTES = {"complex64": 8, "complex128": 16, "float32": 4, "float64": 8}


def _contract(name, labels, ext, dtype="complex64", layout="col", call="async", where="device",
              alpha=(1.0, 0.0), beta=(0.0, 0.0)):
    """labels "la,lb->lc"; ext "a10 b10"; call: "contract" (the reference's
    C += AB wrapper, returns when done), "scaled" (alpha, beta, returns when
    done) or "async" (alpha, beta, queued on the context's stream)."""
    return {"name": name, "kind": "contract", "labels": labels, "ext": ext, "dtype": dtype,
            "layout": layout, "call": call, "where": where, "alpha_re": alpha[0],
            "alpha_im": alpha[1], "beta_re": beta[0], "beta_im": beta[1]}


def _ext(**e):
    return " ".join(f"{k}{v}" for k, v in e.items())


def listed():
    return [
        # The reference's example: one tiny call, all latency.
        _contract("example_10", "abc,bd->acd", _ext(a=10, b=10, c=10, d=10), call="contract"),
        # Drop-in rank-4 contraction with BLAS scalars, column-major.
        _contract("dropin_48", "abcd,efcd->abef", _ext(a=48, b=48, c=48, d=48, e=48, f=48),
                  alpha=(1.0, 0.5), beta=(0.25, 0.0)),
        # Permuted contraction to a small matrix over a long contracted bundle:
        # no operand is a plain matrix.
        _contract("permuted_ec", "abcd,dbea->ec", _ext(a=24, b=32, c=96, d=48, e=64),
                  alpha=(1.0, 0.5), beta=(0.25, 0.0)),
        # The headline product, M = N = K = 4096, device buffers.
        _contract("square_64", "ijkl,klmn->ijmn",
                  _ext(i=64, j=64, k=64, l=64, m=64, n=64)),
        # The same product from and to pinned host memory, copies included.
        _contract("host_64", "ijkl,klmn->ijmn", _ext(i=64, j=64, k=64, l=64, m=64, n=64),
                  call="scaled", where="pinned"),
        # Ragged row-major complex contraction: odd extents, permuted modes.
        _contract("ragged_c64", "abcd,ebfd->aecf", _ext(a=27, b=33, c=35, d=29, e=31, f=37),
                  layout="row", call="contract"),
        # Double-precision complex (chemistry-style accuracy).
        _contract("double_c128", "abcd,efcd->abef", _ext(a=32, b=32, c=32, d=32, e=32, f=32),
                  dtype="complex128", alpha=(1.0, 0.5), beta=(0.25, 0.0)),
        # Real single precision, odd matrix sizes, the reference's real call.
        _contract("ragged_f32", "mk,kn->mn", _ext(m=1999, k=1531, n=2503), dtype="float32",
                  layout="row", call="contract"),
        # Real double precision, a rank-3 tensor times a matrix.
        _contract("tensor_f64", "abc,bd->acd", _ext(a=96, b=96, c=96, d=96), dtype="float64",
                  call="contract"),
        # A tensor-network sweep: updates of uneven bonds as one grouped batch.
        {"name": "sweep_128", "kind": "sweep", "updates": 128, "shapes": 2024, "max_bond": 256},
        # Backward pass of one contraction.
        {"name": "adjoint_32", "kind": "vjp", "labels": "abcd,ebfd->aecf",
         "ext": _ext(a=32, b=32, c=32, d=32, e=32, f=32)},
        # Gradients of a ring of four order-3 tensors, one grouped launch per pass.
        {"name": "ring_64", "kind": "ring", "bond": 64, "phys": 8, "mode": "grouped"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _around(rng, base, lo):
    """An extent of up to `base`, odd or even."""
    return max(lo, min(base, base - rng.randrange(0, max(1, base // 4))))


def draw(rng: random.Random):
    family = rng.randrange(12)
    call = rng.choice(["contract", "async"])
    layout = rng.choice(["col", "row"])
    scal = ((1.0, 0.5), (0.25, 0.0)) if rng.random() < 0.5 else ((1.0, 0.0), (0.0, 0.0))
    if family == 0:
        c = _contract("", "abc,bd->acd", _ext(**{k: rng.randint(2, 24) for k in "abcd"}),
                      dtype=rng.choice(sorted(_TORCH)), layout=layout, call=call)
    elif family == 1:
        b = _log(rng, 8, 48)
        c = _contract("", "abcd,efcd->abef", _ext(**{k: _around(rng, b, 2) for k in "abcdef"}),
                      layout=layout, call="async", alpha=scal[0], beta=scal[1])
    elif family == 2:
        c = _contract("", "abcd,dbea->ec",
                      _ext(a=rng.randint(6, 24), b=rng.randint(8, 32), c=rng.randint(24, 96),
                           d=rng.randint(12, 48), e=rng.randint(16, 64)),
                      layout=layout, call=call if call == "contract" else "async")
    elif family == 3:
        b = _log(rng, 16, 62)
        c = _contract("", "ijkl,klmn->ijmn", _ext(**{k: _around(rng, b, 4) for k in "ijklmn"}),
                      layout=layout, call="async")
    elif family == 4:
        b = rng.randint(20, 60)
        c = _contract("", "ijkl,klmn->ijmn", _ext(**{k: _around(rng, b, 8) for k in "ijklmn"}),
                      layout=layout, call="scaled", where="pinned")
    elif family == 5:
        b = _log(rng, 9, 40)
        c = _contract("", "abcd,ebfd->aecf", _ext(**{k: _around(rng, b, 3) for k in "abcdef"}),
                      layout=layout, call=call)
    elif family == 6:
        b = _log(rng, 6, 32)
        c = _contract("", "abcd,efcd->abef", _ext(**{k: _around(rng, b, 2) for k in "abcdef"}),
                      dtype="complex128", layout=layout, call="async", alpha=scal[0], beta=scal[1])
    elif family == 7:
        c = _contract("", "mk,kn->mn", _ext(**{k: _log(rng, 100, 4000) for k in "mkn"}),
                      dtype="float32", layout=layout, call=call)
    elif family == 8:
        b = _log(rng, 12, 120)
        c = _contract("", "abc,bd->acd", _ext(**{k: _around(rng, b, 3) for k in "abcd"}),
                      dtype="float64", layout=layout, call=call)
    elif family == 9:
        mb = rng.choice([64, 128, 192, 256])
        c = {"kind": "sweep", "updates": _log(rng, 4, 100), "shapes": rng.randrange(1 << 20),
             "max_bond": mb}
    elif family == 10:
        b = _log(rng, 8, 32)
        c = {"kind": "vjp", "labels": "abcd,ebfd->aecf",
             "ext": _ext(**{k: _around(rng, b, 2) for k in "abcdef"})}
    else:
        c = {"kind": "ring", "bond": rng.randint(12, 64), "phys": rng.randint(2, 8),
             "mode": rng.choice(["grouped", "recompute"])}
    c.pop("name", None)
    return c


# ------------------------------------------------------------------ sizes ---

def _parse(case):
    left, lc = case["labels"].split("->")
    la, lb = left.split(",")
    ext = {tok[0]: int(tok[1:]) for tok in case["ext"].split()}
    return la, lb, lc, ext


def _numel(labels, ext):
    return math.prod(ext[ch] for ch in labels)


def _updates(case):
    """(x, y, a, b, s, t) of every sweep update: bonds are multiples of 16."""
    rng = random.Random(case["shapes"])
    bonds = list(range(16, case["max_bond"] + 1, 16))
    return [tuple(rng.choice(bonds) for _ in range(4)) + (rng.choice((2, 4)), rng.choice((2, 4)))
            for _ in range(case["updates"])]


_RING = (["apb", "bpc", "cqd", "dqa"], ["ac", "aqd", ""])


def work(case):
    if case["kind"] in ("contract", "vjp"):
        la, lb, lc, ext = _parse(case)
        na, nb, nc = _numel(la, ext), _numel(lb, ext), _numel(lc, ext)
        full = _numel(set(la) | set(lb), ext)
        if case["kind"] == "vjp":
            # reads A, B, dC; writes dA, dB; two products
            return {"bytes": 8 * (2 * na + 2 * nb + nc), "flops": 16.0 * full}
        es = _BYTES[case["dtype"]]
        cplx = case["dtype"].startswith("complex")
        reads_c = case["call"] == "contract" or case["beta_re"] != 0 or case["beta_im"] != 0
        return {"bytes": es * (na + nb + nc * (2 if reads_c else 1)),
                "flops": (8.0 if cplx else 2.0) * full}
    if case["kind"] == "sweep":
        nbytes = flops = 0
        for x, y, a, b, s, t in _updates(case):
            # reads X1, X2, X3; writes and reads R; writes O
            nbytes += 8 * (x * a * y + a * s * b + y * t * b + 2 * x * s * y * b + x * s * t)
            flops += 8 * x * y * s * b * a + 8 * x * s * t * y * b
        return {"bytes": nbytes, "flops": float(flops)}
    # Ring: three contractions forward, two products for each backward.
    ext = {ch: case["bond"] for ch in "abcd"} | {ch: case["phys"] for ch in "pq"}
    labels, outs = _RING
    cur, flops, nbytes = labels[0], 0.0, 2 * 8 * sum(_numel(x, ext) for x in labels)
    for x, o in zip(labels[1:], outs):
        flops += 3 * 8.0 * _numel(set(cur) | set(x), ext)
        cur = o
    return {"bytes": nbytes, "flops": flops}


# ----------------------------------------------------------------- inputs ---

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(n, dtype, g):
    """Entries (complex: both components) uniform in [-1, 1]."""
    td = _TORCH[dtype]
    real = torch.float32 if dtype in ("complex64", "float32") else torch.float64
    if not td.is_complex:
        return torch.rand(n, device="cuda", generator=g, dtype=real) * 2 - 1
    x = torch.rand(2 * n, device="cuda", generator=g, dtype=real) * 2 - 1
    return torch.view_as_complex(x.view(n, 2))


def _normal(n, std, g):
    x = torch.randn(2 * n, device="cuda", generator=g) * std
    return torch.view_as_complex(x.view(n, 2))


def _inputs(case, seed):
    """The seeded tensors of a case, in device memory."""
    g = _gen(seed)
    if case["kind"] == "contract":
        la, lb, lc, ext = _parse(case)
        return [_uniform(_numel(x, ext), case["dtype"], g) for x in (la, lb, lc)]
    if case["kind"] == "vjp":
        la, lb, lc, ext = _parse(case)
        return [_uniform(_numel(x, ext), "complex64", g).view([ext[ch] for ch in x])
                for x in (la, lb, lc)]
    if case["kind"] == "sweep":
        out = []
        for x, y, a, b, s, t in _updates(case):
            sa, sb = a ** -0.25, b ** -0.25
            out.append((_normal(x * a * y, sa, g).view(x, a, y),
                        _normal(a * s * b, sa, g).view(a, s, b),
                        _normal(y * t * b, sb, g).view(y, t, b)))
        return out
    ext = {ch: case["bond"] for ch in "abcd"} | {ch: case["phys"] for ch in "pq"}
    scale = 1.0 / math.sqrt(case["bond"])
    return [(_uniform(_numel(x, ext), "complex64", g) * scale).view([ext[ch] for ch in x])
            for x in _RING[0]]


_context = None


def _ctx():
    """One context for the program, as a user keeps it."""
    global _context
    if _context is None:
        _context = t1m.Context(0)
    return _context


def _row(z):
    return t1m.tensor(list(z.shape), z, t1m.row_major)


def prepare(case, seed):
    ctx = _ctx()
    if case["kind"] == "contract":
        la, lb, lc, ext = _parse(case)
        xs = _inputs(case, seed)
        if case["where"] == "pinned":
            host = [torch.empty(x.shape, dtype=x.dtype, pin_memory=True) for x in xs]
            for h, x in zip(host, xs):
                h.copy_(x)
            xs = host
        lay = t1m.col_major if case["layout"] == "col" else t1m.row_major
        views = [t1m.tensor([ext[ch] for ch in lab], x, lay) for lab, x in zip((la, lb, lc), xs)]
        alpha = complex(case["alpha_re"], case["alpha_im"])
        beta = complex(case["beta_re"], case["beta_im"])
        if not xs[0].is_complex():
            alpha, beta = alpha.real, beta.real
        state = {"case": case, "ctx": ctx, "labels": (la, lb, lc), "views": views, "c": xs[2],
                 "alpha": alpha, "beta": beta}
    elif case["kind"] == "vjp":
        la, lb, lc, ext = _parse(case)
        a, b, dc = _inputs(case, seed)
        da, db = torch.empty_like(a), torch.empty_like(b)
        state = {"case": case, "ctx": ctx, "labels": (la, lb, lc),
                 "views": [_row(z) for z in (a, b, dc, da, db)], "grads": [da, db]}
    elif case["kind"] == "sweep":
        ups, xs = _updates(case), _inputs(case, seed)
        nr = [x * s * y * b for x, y, a, b, s, t in ups]
        no = [x * s * t for x, y, a, b, s, t in ups]
        r_all = torch.empty(sum(nr), dtype=torch.complex64, device="cuda")
        o_all = torch.empty(sum(no), dtype=torch.complex64, device="cuda")
        items = []
        for (x, y, a, b, s, t), (x1, x2, x3), r, o in zip(ups, xs, r_all.split(nr),
                                                          o_all.split(no)):
            first = len(items)
            r, o = r.view(x, s, y, b), o.view(x, s, t)
            items.append((1.0, _row(x1), "xay", _row(x2), "asb", 0.0, _row(r), "xsyb", -1))
            items.append((1.0, _row(r), "xsyb", _row(x3), "ytb", 0.0, _row(o), "xst", first))
        torch.cuda.synchronize()
        state = {"case": case, "ctx": ctx, "group": t1m.Group(items, ctx=ctx, graph=True),
                 "out": [r_all, o_all], "keep": xs}
    else:
        xs = _inputs(case, seed)
        chain = ContractionChain(*_RING, mode=case["mode"])
        state = {"case": case, "ctx": ctx, "chain": chain, "xs": xs,
                 "one": torch.ones((), dtype=torch.complex64, device="cuda")}
    torch.cuda.synchronize()  # the context has a stream of its own
    return state


def run(state):
    case, ctx = state["case"], state["ctx"]
    if case["kind"] == "contract":
        (a, b, c), (la, lb, lc) = state["views"], state["labels"]
        if case["call"] == "contract":
            if case["dtype"].startswith("complex"):
                t1m.contract(a, la, b, lb, c, lc, ctx=ctx)
            else:
                t1m.contract(1.0, a, la, b, lb, 1.0, c, lc, ctx=ctx)
        elif case["call"] == "scaled":
            t1m.contract_scaled(state["alpha"], a, la, b, lb, state["beta"], c, lc, ctx=ctx)
        else:
            t1m.contract_raw(state["alpha"], a, la, b, lb, state["beta"], c, lc,
                             t1m.FLAG_NO_TIMING, ctx)
        return state["c"]
    if case["kind"] == "vjp":
        (a, b, dc, da, db), (la, lb, lc) = state["views"], state["labels"]
        t1m.contract_vjp(dc, lc, a, la, b, lb, da, db, ctx=ctx, timed=False)
        return state["grads"]
    if case["kind"] == "sweep":
        state["group"].launch(timed=False)
        return state["out"]
    return state["chain"].backward(state["xs"], state["one"], ctx=ctx)


# ------------------------------------------------------------------ exact ---

def _wide(x):
    return x.to(torch.complex128 if x.is_complex() else torch.float64)


def exact(case, seed):
    xs = _inputs(case, seed)
    if case["kind"] == "contract":
        la, lb, lc, ext = _parse(case)
        a, b, c = (_wide(x) for x in xs)
        shape = [[ext[ch] for ch in lab] for lab in (la, lb, lc)]
        if case["layout"] == "col":
            # A column-major buffer is the row-major one of the reversed modes.
            la, lb, lc = la[::-1], lb[::-1], lc[::-1]
            shape = [s[::-1] for s in shape]
        ab = torch.einsum(f"{la},{lb}->{lc}", a.view(shape[0]), b.view(shape[1])).reshape(-1)
        if case["call"] == "contract":
            return c + ab
        alpha = complex(case["alpha_re"], case["alpha_im"])
        beta = complex(case["beta_re"], case["beta_im"])
        if not ab.is_complex():
            alpha, beta = alpha.real, beta.real
        return alpha * ab + beta * c
    if case["kind"] == "vjp":
        la, lb, lc, _ = _parse(case)
        a, b, dc = (_wide(x) for x in xs)
        return [torch.einsum(f"{lc},{lb}->{la}", dc, b.conj()),
                torch.einsum(f"{la},{lc}->{lb}", a.conj(), dc)]
    if case["kind"] == "sweep":
        rs, os_ = [], []
        for x1, x2, x3 in xs:
            r = torch.einsum("xay,asb->xsyb", _wide(x1), _wide(x2))
            os_.append(torch.einsum("xsyb,ytb->xst", r, _wide(x3)).reshape(-1))
            rs.append(r.reshape(-1))
        return [torch.cat(rs), torch.cat(os_)]
    labels, _ = _RING
    ws = [_wide(x).requires_grad_() for x in xs]
    y = torch.einsum(",".join(labels) + "->", *ws)
    # d Re(y) in the conjugate-Wirtinger convention, for an upstream gradient 1.
    return list(torch.autograd.grad(y.real, ws))
