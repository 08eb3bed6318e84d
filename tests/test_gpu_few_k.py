"""Float64 products over few k, whose large outputs take the plain kernel's
128 x 64 tile and whose small ones 16 x 16 and 8 x 8 tiles: one chain of FMAs
in the order of k whichever tile it is, so the bits are those of the same
chain computed on the host with exact products (integers), and the same for
an output and a part of it (gpu)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["row", "col"])
@pytest.mark.parametrize("k", [1, 3, 7, 8, 9])
@pytest.mark.parametrize("mn", [(1000, 1000), (1025, 511), (129, 6000), (40, 30)],
                         ids=lambda s: "x".join(map(str, s)))
def test_few_k(ctx, torch_cuda, mn, k, layout):
    import t1m_gb300 as t1m
    torch = torch_cuda
    m, n = mn
    rng = np.random.default_rng(80)
    order, L = ("C", t1m.row_major) if layout == "row" else ("F", t1m.col_major)

    def run(a, b, c, beta):
        bufs = [torch.from_numpy(np.ravel(x, order=order).copy()).cuda() for x in (a, b, c)]
        v = [t1m.tensor(list(x.shape), g, L) for x, g in zip((a, b, c), bufs)]
        t1m.contract_scaled(2.0, v[0], "mk", v[1], "kn", beta, v[2], "mn", ctx=ctx)
        torch.cuda.synchronize()
        return bufs[2].cpu().numpy().reshape(c.shape, order=order)

    a, b, c = (rng.integers(-1000, 1000, s).astype(np.float64) for s in ((m, k), (k, n), (m, n)))
    np.testing.assert_array_equal(run(a, b, c, 0.5), 2.0 * (a @ b) + 0.5 * c)
    a, b, c = (rng.uniform(-1, 1, s) for s in ((m, k), (k, n), (m, n)))
    whole = run(a, b, c, 0.0)
    if k <= 8:
        np.testing.assert_array_equal(whole[:24, :24], run(a[:24], b[:, :24], c[:24, :24], 0.0))
    ref = 2.0 * np.einsum("mk,kn->mn", a.astype(np.longdouble), b.astype(np.longdouble))
    assert np.abs(whole - ref).max() <= 2 * (k + 1) * 2.0**-53 * k
