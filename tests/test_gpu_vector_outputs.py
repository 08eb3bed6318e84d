"""Contractions to vectors and thin matrices over long bundles (complex64,
float32): the K ranges' partial products start at odd element offsets, so
their stores may not be wider than an element.  Both layouts, either operand
the vector, the adjoint and batch labels, against FP64: the automatic
method's bound of 1e-6 of the largest output.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(17, 1, 16384), (33, 1, 8192), (101, 1, 4096), (4095, 1, 1024), (1999, 1, 1531),
         (1, 17, 16384), (1, 33, 70000), (1, 101, 4096), (1, 145, 8192), (3, 33, 4096),
         (33, 3, 4096)]


def _rand(rng, shape, dtype):
    x = rng.uniform(-1, 1, shape)
    return (x + 1j * rng.uniform(-1, 1, shape) if dtype == np.complex64 else x).astype(dtype)


def _wide(x):
    return x.astype(np.complex128 if np.iscomplexobj(x) else np.float64)


@pytest.mark.parametrize("dtype", [np.complex64, np.float32])
@pytest.mark.parametrize("method", ["auto", "tc_3xtf32", "tc_bf16x6"])
@pytest.mark.parametrize("layout", ["row", "col"])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
def test_vector_outputs(ctx, torch_cuda, size, layout, method, dtype):
    import t1m_gb300 as t1m
    m, n, k = size
    rng = np.random.default_rng(7)
    A, B, C = (_rand(rng, s, dtype) for s in ((m, k), (k, n), (m, n)))
    order, L = ("C", t1m.row_major) if layout == "row" else ("F", t1m.col_major)
    if n == 1:
        labels, ops = ("mk", "k", "m"), (A, B[:, 0], C[:, 0])
    elif m == 1:
        labels, ops = ("k", "kn", "n"), (A[0], B, C[0])
    else:
        labels, ops = ("mk", "kn", "mn"), (A, B, C)
    bufs = [torch_cuda.from_numpy(np.ravel(x, order=order).copy()).cuda() for x in ops]
    a, b, c = (t1m.tensor(list(x.shape), g, L) for x, g in zip(ops, bufs))
    ctx.set_method(method)
    try:
        t1m.contract_scaled(1.5, a, labels[0], b, labels[1], 0.25, c, labels[2], ctx=ctx)
    finally:
        ctx.set_method("auto")
    torch_cuda.cuda.synchronize()
    ref = 1.5 * (_wide(A) @ _wide(B)) + 0.25 * _wide(C)
    got = bufs[2].cpu().numpy().reshape(ops[2].shape, order=order).reshape(m, n)
    assert np.abs(got - ref).max() <= 1e-6 * np.abs(ref).max()


@pytest.mark.parametrize("m,k", [(101, 4096), (4095, 1024)])
def test_vector_output_adjoint(ctx, torch_cuda, m, k):
    """dA = dy x^H and dx = A^H dy of y = A x: an outer product and a vector
    over m."""
    import t1m_gb300 as t1m
    rng = np.random.default_rng(8)
    A, x, dy = (_rand(rng, s, np.complex64) for s in ((m, k), (k,), (m,)))
    g = [torch_cuda.from_numpy(z).cuda() for z in (A, x, dy)]
    dA, dx = torch_cuda.empty_like(g[0]), torch_cuda.empty_like(g[1])
    v = lambda z: t1m.tensor(list(z.shape), z, t1m.row_major)  # noqa: E731
    t1m.contract_vjp(v(g[2]), "m", v(g[0]), "mk", v(g[1]), "k", v(dA), v(dx), ctx=ctx)
    torch_cuda.cuda.synchronize()
    A, x, dy = _wide(A), _wide(x), _wide(dy)
    for got, ref in ((dA, np.outer(dy, x.conj())), (dx, A.conj().T @ dy)):
        assert np.abs(got.cpu().numpy() - ref).max() <= 1e-6 * np.abs(ref).max()


@pytest.mark.parametrize("m", [17, 101])
def test_vector_output_batched(ctx, torch_cuda, m):
    """Batch labels: each batch index is a product of its own, with C (and its
    partials) at odd offsets."""
    import t1m_gb300 as t1m
    rng = np.random.default_rng(9)
    A, x = _rand(rng, (3, m, 20000), np.complex64), _rand(rng, (3, 20000), np.complex64)
    ga, gx = (torch_cuda.from_numpy(z).cuda() for z in (A, x))
    gy = torch_cuda.zeros((3, m), dtype=torch_cuda.complex64, device="cuda")
    v = lambda z: t1m.tensor(list(z.shape), z, t1m.row_major)  # noqa: E731
    t1m.contract_scaled(1.0, v(ga), "bmk", v(gx), "bk", 0.0, v(gy), "bm", ctx=ctx)
    torch_cuda.cuda.synchronize()
    ref = np.einsum("bmk,bk->bm", _wide(A), _wide(x))
    assert np.abs(gy.cpu().numpy() - ref).max() <= 1e-6 * np.abs(ref).max()
