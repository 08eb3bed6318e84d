"""Which form the items of a grouped launch take, seen in their bits (gpu)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _items(t1m, torch, rng, shapes, dtype=np.complex64):
    items, keep, outs = [], [], []
    for m, n, k in shapes:
        def rand(s):
            x = rng.uniform(-1, 1, s)
            return (x + 1j * rng.uniform(-1, 1, s) if np.issubdtype(dtype, np.complexfloating)
                    else x).astype(dtype)
        a, b = rand((m, k)), rand((k, n))
        g = [torch.from_numpy(x).cuda() for x in (a, b, np.zeros((m, n), dtype))]
        v = [t1m.tensor(list(x.shape), x, t1m.row_major) for x in g]
        items.append((1.0, v[0], "mk", v[1], "kn", 0.0, v[2], "mn", -1))
        keep.append((a, b))
        outs.append(g)
    torch.cuda.synchronize()
    return items, keep, outs


@pytest.mark.parametrize("count", [1, 8])
@pytest.mark.parametrize("size", [(200, 100, 300), (64, 64, 512), (512, 256, 256), (65, 33, 1024)],
                         ids=lambda s: "x".join(map(str, s)))
def test_tensor_core_batch_is_not_split(ctx, torch_cuda, size, count):
    """A batch of tensor-core items only is one persistent launch, its items
    unsplit up to K = 1024: the bits of the same launch asked for by option."""
    import t1m_gb300 as t1m
    torch = torch_cuda
    items, keep, outs = _items(t1m, torch, np.random.default_rng(70), [size] * count)
    got = []
    for options in (0, t1m.GROUP_ONE_LAUNCH | t1m.GROUP_TILE_128):
        g = t1m.Group(items, ctx=ctx, graph=False, options=options)
        rep = g.launch()
        torch.cuda.synchronize()
        assert rep.kernels == 1
        got.append([x[2].cpu().numpy().copy() for x in outs])
        for x in outs:
            x[2].zero_()
        torch.cuda.synchronize()
        g.close()
    for x, y, (a, b) in zip(*got, keep):
        np.testing.assert_array_equal(x, y)
        ref = a.astype(np.complex128) @ b.astype(np.complex128)
        assert np.abs(x - ref).max() <= 1e-6 * np.abs(ref).max()


@pytest.mark.parametrize("count", [1, 8, 80])
@pytest.mark.parametrize("dtype", [np.complex64, np.float64])
def test_skinny_rows_per_block(ctx, torch_cuda, dtype, count):
    """Items of a few columns around the 256 rows from which a block may take
    128 of them: few items in blocks of 32 rows, many in tall ones."""
    import t1m_gb300 as t1m
    torch = torch_cuda
    shapes = [((255, 256, 257, 383, 1000)[i % 5], 1 + i % 4, 500 + 2 * i) for i in range(count)]
    items, keep, outs = _items(t1m, torch, np.random.default_rng(71), shapes, dtype)
    g = t1m.Group(items, ctx=ctx, graph=False)
    g.launch()
    torch.cuda.synchronize()
    for (a, b), out in zip(keep, outs):
        ref = a.astype(np.complex128) @ b.astype(np.complex128)
        bound = 1e-6 if dtype == np.complex64 else 1e-13
        assert np.abs(out[2].cpu().numpy() - ref).max() <= bound * np.abs(ref).max()
