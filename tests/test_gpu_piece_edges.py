"""Products over operand pieces at the edges of their tiles (pairs of 128
complex or 256 real rows, widths of 32 to 256 columns), 32-k stages, 16-k MMA
steps and split passes, with the operands in every read order (rows, K, a
later K mode) and exchanged or not, against FP64: BF16x6's bound of 1e-6 of
the largest output.  Where both operands also load by TMA, the
CTA-pair form gives the same bits.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (labels, extents): plain matrices with ragged M, N, K; permuted modes whose
# K runs are a first mode, no mode, or a later mode of the plan's K order.
CASES = [
    ("mk,kn->mn", dict(m=129, k=17, n=161)),
    ("mk,kn->mn", dict(m=200, k=33, n=385)),
    ("mk,kn->mn", dict(m=300, k=260, n=130)),
    ("mk,nk->mn", dict(m=513, k=48, n=97)),
    ("mk,kn->nm", dict(m=257, k=129, n=255)),
    ("abcd,ebfd->aecf", dict(a=13, b=9, c=15, d=7, e=17, f=11)),
    ("abcd,ebfd->aecf", dict(a=16, b=16, c=16, d=16, e=16, f=16)),
    ("apqb,cqpd->abcd", dict(a=16, b=16, p=32, q=10, c=15, d=14)),
    ("apqb,cqpd->cdab", dict(a=17, b=15, p=6, q=33, c=14, d=15)),
]


def _tensor(rng, labels, ext, dt):
    s = [ext[ch] for ch in labels]
    x = rng.uniform(-1, 1, s)
    return (x + 1j * rng.uniform(-1, 1, s) if dt == np.complex64 else x).astype(dt)


def _run(ctx, torch, labels, ts, layout, form, beta):
    import t1m_gb300 as t1m
    order = "C" if layout == "row" else "F"
    L = t1m.row_major if layout == "row" else t1m.col_major
    bufs = [torch.from_numpy(np.ravel(x, order=order).copy()).cuda() for x in ts]
    a, b, c = (t1m.tensor(list(x.shape), g, L) for x, g in zip(ts, bufs))
    la, rest = labels.split(",")
    lb, lc = rest.split("->")
    ctx.set_tile_form(form)
    ctx.set_method("tc_bf16x6")  # the automatic method runs the smallest cases plain
    try:
        rep = t1m.contract_scaled(0.5, a, la, b, lb, beta, c, lc, ctx=ctx)
    finally:
        ctx.set_tile_form("auto")
        ctx.set_method("auto")
    torch.cuda.synchronize()
    return bufs[2].cpu().numpy().reshape(ts[2].shape, order=order), rep


@pytest.mark.parametrize("beta", [0.0, 0.25])
@pytest.mark.parametrize("layout", ["row", "col"])
@pytest.mark.parametrize("dt", [np.complex64, np.float32])
@pytest.mark.parametrize("case", CASES, ids=lambda c: c[0] + "-" + "x".join(map(str, c[1].values())))
def test_piece_edges(ctx, torch_cuda, case, dt, layout, beta):
    labels, ext = case
    rng = np.random.default_rng(77)
    la, rest = labels.split(",")
    lb, lc = rest.split("->")
    ts = [_tensor(rng, x, ext, dt) for x in (la, lb, lc)]
    wide = np.complex128 if dt == np.complex64 else np.float64
    ref = 0.5 * np.einsum(labels, ts[0].astype(wide), ts[1].astype(wide)) + beta * ts[2]
    got, rep = _run(ctx, torch_cuda, labels, ts, layout, "auto", beta)
    assert rep.method == 4 and rep.fetch["pieces"], rep.fetch
    assert np.abs(got - ref).max() <= 1e-6 * np.abs(ref).max()
    pair, rp = _run(ctx, torch_cuda, labels, ts, layout, "pair", beta)
    if rp.method == rep.method and rp.split_k == rep.split_k and rp.fetch["pair"]:
        np.testing.assert_array_equal(got, pair)


@pytest.mark.parametrize("mn", [(150, 1900), (1900, 150)])
@pytest.mark.parametrize("layout", ["row", "col"])
def test_pieces_workspace_of_exchanged_operands(built_lib, torch_cuda, layout, mn):
    """The first product of a context (no larger workspace left from an earlier
    one), far from square: the pieces of whichever operand takes the 1M rows
    fit the workspace."""
    import t1m_gb300 as t1m
    ctx = t1m.Context()
    rng = np.random.default_rng(78)
    ext = dict(m=mn[0], n=mn[1], k=300)
    ts = [_tensor(rng, x, ext, np.complex64) for x in ("mk", "kn", "mn")]
    got, rep = _run(ctx, torch_cuda, "mk,kn->mn", ts, layout, "auto", 0.25)
    ctx.close()
    assert rep.fetch["pieces"]
    ref = 0.5 * ts[0].astype(np.complex128) @ ts[1].astype(np.complex128) + 0.25 * ts[2]
    assert np.abs(got - ref).max() <= 1e-6 * np.abs(ref).max()
