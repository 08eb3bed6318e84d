"""Products queued back to back, each reading what the one before it wrote as
its first or second operand: kernels start before the ones ahead of them have
ended (dependent launches), so the results must be those of the same products
with a wait after each, bit for bit (gpu)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("second", [False, True])
@pytest.mark.parametrize("layout", ["row", "col"])
@pytest.mark.parametrize("e", [16, 23, 32])
def test_back_to_back(ctx, torch_cuda, e, layout, second):
    import t1m_gb300 as t1m
    torch = torch_cuda
    rng = np.random.default_rng(64)
    n, dims = e ** 4, [e] * 4
    L = t1m.col_major if layout == "col" else t1m.row_major

    def rand():
        x = rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n)
        return torch.from_numpy((x / e).astype(np.complex64)).cuda()

    a, start = rand(), rand()
    steps = 12

    def run(wait):
        outs = [start] + [torch.zeros_like(a) for _ in range(steps)]
        torch.cuda.synchronize()
        v = [t1m.tensor(dims, x, L) for x in outs]
        other = t1m.tensor(dims, a, L)
        for x, y in zip(v, v[1:]):
            ops = (other, x) if second else (x, other)
            t1m.contract_raw(1.0, ops[0], "abcd", ops[1], "ebfd", 0.0, y, "aecf",
                             t1m.FLAG_NO_TIMING, ctx)
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return outs

    want = run(True)
    for _ in range(3):
        for got, ref in zip(run(False), want):
            assert torch.equal(torch.view_as_real(got), torch.view_as_real(ref))


def test_two_contexts_interleaved(ctx, torch_cuda):
    """Two contexts on streams of their own, their calls interleaved."""
    import t1m_gb300 as t1m
    torch = torch_cuda
    rng = np.random.default_rng(65)

    def rand(*s):
        return torch.from_numpy((rng.uniform(-1, 1, s) + 1j * rng.uniform(-1, 1, s))
                                .astype(np.complex64)).cuda()

    v = lambda z: t1m.tensor(list(z.shape), z, t1m.row_major)  # noqa: E731
    a, b = rand(20, 22, 24, 26), rand(18, 22, 21, 26)     # over pieces
    x, y = rand(50, 4096), rand(4096, 40)                 # streamed
    c = [torch.zeros((20, 18, 24, 21), dtype=torch.complex64, device="cuda") for _ in range(2)]
    d = [torch.zeros((50, 40), dtype=torch.complex64, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    other = t1m.Context(0)
    for i in range(40):
        for w in (ctx, other) if i % 2 else (other, ctx):
            slot = 0 if w is ctx else 1
            t1m.contract_raw(1.0, v(a), "abcd", v(b), "ebfd", 0.0, v(c[slot]), "aecf",
                             t1m.FLAG_NO_TIMING, w)
            t1m.contract_raw(1.0, v(x), "mk", v(y), "kn", 0.0, v(d[slot]), "mn",
                             t1m.FLAG_NO_TIMING, w)
    torch.cuda.synchronize()
    other.close()
    for p in (c, d):
        assert torch.equal(torch.view_as_real(p[0]), torch.view_as_real(p[1]))
    w = a.to(torch.complex128), b.to(torch.complex128)
    ref = torch.einsum("abcd,ebfd->aecf", *w)
    assert (c[0] - ref).abs().max() <= 1e-6 * ref.abs().max()
