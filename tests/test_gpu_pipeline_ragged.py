"""Host buffers whose halves and slabs do not fill the tiles of the product
over operand pieces (the last half or slab ends inside a tile and inside a
group of eight rows): the same bits as from device buffers (gpu)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["col", "row"])
@pytest.mark.parametrize("dtype,m,n,k", [(np.complex64, 2080, 2200, 2050),
                                         (np.complex64, 1991, 2305, 2049),
                                         (np.float32, 4160, 2200, 4100),
                                         (np.float32, 2201, 4227, 4097)])
def test_ragged_host_equals_device(ctx, torch_cuda, dtype, m, n, k, layout):
    import t1m_gb300 as t1m
    rng = np.random.default_rng(63)

    def rand(size):
        x = rng.uniform(-1, 1, size)
        return (x + 1j * rng.uniform(-1, 1, size) if dtype == np.complex64 else x).astype(dtype)

    L = t1m.col_major if layout == "col" else t1m.row_major
    A, B, C = rand(m * k), rand(k * n), np.zeros(m * n, dtype)
    dev = [torch_cuda.from_numpy(x.copy()).cuda() for x in (A, B, C)]
    reps = [t1m.contract_scaled(1.0, t1m.tensor([m, k], a, L), "mk", t1m.tensor([k, n], b, L), "kn",
                                0.0, t1m.tensor([m, n], c, L), "mn", ctx=ctx)
            for a, b, c in ((A, B, C), dev)]
    torch_cuda.cuda.synchronize()
    assert reps[0].kernels > reps[1].kernels and all(r.fetch["pieces"] for r in reps)
    np.testing.assert_array_equal(C, dev[2].cpu().numpy())
