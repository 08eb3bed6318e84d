"""The small output tiles (small_tile.cu) of the plain method at the edges of
the 16 x 16 and 8 x 8 tiles, the 16-k stages and the k slices, split and
unsplit, against an extended-precision product.  Elementwise bound: a sum of K
products in any order differs from the exact one by at most about (4 K + 8) u
|A||B| (four real products per complex term), u = 2^-53 or 2^-24.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (8, 8, 16), (9, 7, 17), (16, 16, 15), (17, 33, 47), (31, 5, 130),
          (96, 80, 64), (250, 19, 3), (40, 40, 1000), (300, 290, 33)]


@pytest.mark.parametrize("splits", [0, 3])
@pytest.mark.parametrize("layout", ["row", "col"])
@pytest.mark.parametrize("dt", [np.float64, np.complex128, np.float32, np.complex64])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_small_tile_edges(ctx, torch_cuda, shape, dt, layout, splits):
    import t1m_gb300 as t1m
    torch = torch_cuda
    M, N, K = shape
    rng = np.random.default_rng(M + N + K)

    def rand(*s):
        x = rng.uniform(-1, 1, s)
        return (x + 1j * rng.uniform(-1, 1, s) if conj else x).astype(dt)

    conj = np.dtype(dt).kind == "c"

    A, B, C = rand(M, K), rand(K, N), rand(M, N)
    order = "C" if layout == "row" else "F"
    L = t1m.row_major if layout == "row" else t1m.col_major
    alpha, beta = (0.5 - 1j, 0.25) if conj else (0.5, 0.25)
    ga, gb, gc = (torch.from_numpy(np.ravel(x, order=order).copy()).cuda() for x in (A, B, C))
    ctx.set_method("plain")
    ctx.set_split_k(splits)
    try:
        t1m.contract_scaled(alpha, t1m.tensor([M, K], ga, L), "mk", t1m.tensor([K, N], gb, L),
                            "kn", beta, t1m.tensor([M, N], gc, L), "mn", ctx=ctx, conj_a=conj)
    finally:
        ctx.set_split_k(0)
        ctx.set_method("auto")
    torch.cuda.synchronize()
    wide = np.clongdouble if conj else np.longdouble
    Aw = np.conj(A) if conj else A
    ref = wide(alpha) * (Aw.astype(wide) @ B.astype(wide)) + wide(beta) * C.astype(wide)
    got = gc.cpu().numpy().reshape((M, N), order=order)
    bound = (4 * K + 8) * np.finfo(dt).eps / 2 * (abs(alpha) * (abs(A) @ abs(B)) * 2 + abs(beta) * abs(C) * 2)
    assert np.all(np.abs(got - ref.astype(dt)) <= bound)


@pytest.mark.parametrize("mn", [80, 256])
@pytest.mark.parametrize("K", [2, 3, 4, 5, 6, 9])
@pytest.mark.parametrize("dt", [np.float64, np.float32])
def test_few_terms_round_like_one_chain(ctx, torch_cuda, dt, K, mn):
    """Outputs of few terms round no more than one FMA chain (rms; the chain
    is evaluated with one rounding per term, 5% allowed for the sample)."""
    import t1m_gb300 as t1m
    torch = torch_cuda
    rng = np.random.default_rng(K + mn)
    A, B = (rng.uniform(-1, 1, s).astype(dt) for s in ((mn, K), (K, mn)))
    wide = np.longdouble
    chain = np.zeros((mn, mn), dt)
    for k in range(K):
        chain = (A[:, k:k + 1].astype(wide) * B[k].astype(wide) + chain.astype(wide)).astype(dt)
    exact = A.astype(wide) @ B.astype(wide)
    ga, gb = torch.from_numpy(A.ravel()).cuda(), torch.from_numpy(B.ravel()).cuda()
    gc = torch.zeros(mn * mn, dtype=ga.dtype, device="cuda")
    row = t1m.row_major
    t1m.contract_scaled(1.0, t1m.tensor([mn, K], ga, row), "mk", t1m.tensor([K, mn], gb, row),
                        "kn", 0.0, t1m.tensor([mn, mn], gc, row), "mn", ctx=ctx)
    torch.cuda.synchronize()
    got = gc.cpu().numpy().reshape(mn, mn)
    rms = lambda x: float(np.sqrt(np.mean((x.astype(wide) - exact) ** 2)))
    assert rms(got) <= 1.05 * rms(chain)


@pytest.mark.parametrize("mn", [24, 256])
@pytest.mark.parametrize("dt", [np.float32, np.complex64])
def test_infinite_sums_stay_infinite(ctx, torch_cuda, dt, mn):
    """Infinite, overflowing and NaN sums of the joined chains."""
    import t1m_gb300 as t1m
    torch = torch_cuda
    K = 8
    A, B = np.ones((mn, K), dt), np.ones((K, mn), dt)
    A[0, 1] = np.inf                     # an infinite term
    A[1, :] = np.finfo(np.float32).max   # overflow in the additions
    A[2, 3] = np.nan
    ga, gb = torch.from_numpy(A.ravel()).cuda(), torch.from_numpy(B.ravel()).cuda()
    gc = torch.zeros(mn * mn, dtype=ga.dtype, device="cuda")
    row = t1m.row_major
    ctx.set_method("plain")
    try:
        t1m.contract_scaled(1.0, t1m.tensor([mn, K], ga, row), "mk", t1m.tensor([K, mn], gb, row),
                            "kn", 0.0, t1m.tensor([mn, mn], gc, row), "mn", ctx=ctx)
    finally:
        ctx.set_method("auto")
    torch.cuda.synchronize()
    got = gc.cpu().numpy().reshape(mn, mn).real
    if dt is np.float32:
        assert np.all(np.isposinf(got[:2]))
    else:
        assert np.all(np.isposinf(got[1]))
    assert np.all(np.isnan(got[2])) and np.all(got[3:] == K)
