"""Streamed products (small complex64 outputs over long contracted bundles) at
the edges of their 64-row and 128-column tiles, 32-k stages and K ranges, with
each operand read along its rows, along K, or along different K modes of the
two (interleaved K order), conjugated and not, against FP64: the automatic
method's bound of 1e-6 of the largest output.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    ("mk,kn->mn", dict(m=1, k=70000, n=9)),
    ("mk,kn->mn", dict(m=64, k=1024, n=128)),
    ("mk,kn->mn", dict(m=65, k=4097, n=63)),
    ("mk,nk->mn", dict(m=130, k=3001, n=20)),
    ("km,kn->nm", dict(m=17, k=2050, n=257)),
    ("abcd,dbea->ec", dict(a=8, b=9, c=33, d=16, e=40)),
    ("abcd,dbea->ec", dict(a=12, b=10, c=17, d=24, e=66)),
    ("abcd,dbea->ec", dict(a=7, b=11, c=20, d=23, e=18)),
]


@pytest.mark.parametrize("flags", [0, 6])
@pytest.mark.parametrize("layout", ["row", "col"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: c[0] + "-" + "x".join(map(str, c[1].values())))
def test_stream_edges(ctx, torch_cuda, case, layout, flags):
    import t1m_gb300 as t1m
    labels, ext = case
    la, rest = labels.split(",")
    lb, lc = rest.split("->")
    rng = np.random.default_rng(91)

    def rand(lab):
        s = [ext[ch] for ch in lab]
        return (rng.uniform(-1, 1, s) + 1j * rng.uniform(-1, 1, s)).astype(np.complex64)

    ts = [rand(x) for x in (la, lb, lc)]
    order = "C" if layout == "row" else "F"
    L = t1m.row_major if layout == "row" else t1m.col_major
    bufs = [torch_cuda.from_numpy(np.ravel(x, order=order).copy()).cuda() for x in ts]
    a, b, c = (t1m.tensor(list(x.shape), g, L) for x, g in zip(ts, bufs))
    alpha, beta = 1 - 0.5j, 0.25
    rep = t1m.contract_scaled(alpha, a, la, b, lb, beta, c, lc, ctx=ctx, conj_a=bool(flags & 2),
                              conj_b=bool(flags & 4))
    torch_cuda.cuda.synchronize()
    assert rep.method == 4 and rep.fetch["a"] == "gather" and not rep.fetch["pieces"], rep.fetch
    A, B = (x.astype(np.complex128) for x in ts[:2])
    A, B = (np.conj(A) if flags & 2 else A), (np.conj(B) if flags & 4 else B)
    ref = alpha * np.einsum(labels, A, B) + beta * ts[2]
    got = bufs[2].cpu().numpy().reshape(ts[2].shape, order=order)
    assert np.abs(got - ref).max() <= 1e-6 * np.abs(ref).max()
