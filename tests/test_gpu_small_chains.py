"""Small FP32 products over more than 32 k sum eight chains of every eighth k
on the plain kernel, joined without loss: 2^24 in one chain and two 1s in
another give 2^24 + 2 exactly, which any order with the 1s in the first chain
rounds to 2^24 (gpu)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mn", [(3, 5), (8, 8), (40, 48), (130, 70)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("k", [33, 48])
@pytest.mark.parametrize("dtype", [np.float32, np.complex64])
def test_small_product_chains(ctx, torch_cuda, dtype, k, mn):
    import t1m_gb300 as t1m
    torch = torch_cuda
    m, n = mn
    row = np.zeros(k)
    row[[0, 4, 12]] = 2.0**24, 1, 1
    for shift in range(4):  # chains 0 and 4, 1 and 5, ...
        a = np.broadcast_to(np.roll(row, shift), (m, k)).astype(dtype)
        g = [torch.from_numpy(np.ascontiguousarray(x)).cuda()
             for x in (a, np.ones((k, n), dtype), np.zeros((m, n), dtype))]
        v = [t1m.tensor(list(x.shape), x, t1m.row_major) for x in g]
        ctx.set_method("plain")
        ctx.set_split_k(1)
        try:
            t1m.contract_scaled(1.0, v[0], "mk", v[1], "kn", 0.0, v[2], "mn", ctx=ctx)
        finally:
            ctx.set_split_k(0)
            ctx.set_method("auto")
        torch.cuda.synchronize()
        np.testing.assert_array_equal(g[2].cpu().numpy(), np.full((m, n), 2.0**24 + 2, dtype))
