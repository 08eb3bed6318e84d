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
