"""Small FP32 products on the plain kernel sum eight chains of every eighth k,
joined without loss: 2^24 in one chain and two 1s in another give 2^24 + 2
exactly, which any order with the 1s in the first chain rounds to 2^24 (gpu)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mn", [(3, 5), (8, 8), (40, 48), (130, 70)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("dtype", [np.float32, np.complex64])
def test_small_product_chains(ctx, torch_cuda, dtype, mn):
    import t1m_gb300 as t1m
    torch = torch_cuda
    m, n = mn
    row = np.zeros(16)
    row[[0, 4, 12]] = 2.0**24, 1, 1
    for shift in range(4):  # chains 0 and 4, 1 and 5, ...
        a = np.broadcast_to(np.roll(row, shift), (m, 16)).astype(dtype)
        g = [torch.from_numpy(np.ascontiguousarray(x)).cuda()
             for x in (a, np.ones((16, n), dtype), np.zeros((m, n), dtype))]
        v = [t1m.tensor(list(x.shape), x, t1m.row_major) for x in g]
        ctx.set_method("plain")
        try:
            t1m.contract_scaled(1.0, v[0], "mk", v[1], "kn", 0.0, v[2], "mn", ctx=ctx)
        finally:
            ctx.set_method("auto")
        torch.cuda.synchronize()
        np.testing.assert_array_equal(g[2].cpu().numpy(), np.full((m, n), 2.0**24 + 2, dtype))
