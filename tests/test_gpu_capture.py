"""Queued calls captured in a caller's CUDA graph, after one call has made the
plans and workspaces: every form's kernels (some of which start before the
ones ahead of them have ended) replay on new inputs with the bits of plain
calls (gpu)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    ("mk,kn->mn", dict(m=512, k=384, n=640), np.complex64),          # pieces, one split pass
    ("abcd,ebfd->aecf", dict(a=14, b=16, c=18, d=12, e=15, f=17), np.complex64),  # two passes
    ("abcd,dbea->ec", dict(a=8, b=16, c=40, d=24, e=33), np.complex64),           # streamed
    ("mk,k->m", dict(m=101, k=4096), np.complex64),                  # streamed vector
    ("abc,bd->acd", dict(a=10, b=10, c=10, d=10), np.complex64),     # small tiles
    ("abc,bd->acd", dict(a=40, b=50, c=30, d=20), np.float64),
    ("mk,kn->mn", dict(m=1001, k=803, n=905), np.float32),           # real pieces
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: c[0] + "-" + np.dtype(c[2]).name)
def test_captured_calls(built_lib, torch_cuda, case):
    import t1m_gb300 as t1m
    torch = torch_cuda
    labels, ext, dtype = case
    la, rest = labels.split(",")
    lb, lc = rest.split("->")
    rng = np.random.default_rng(90)

    def rand(lab):
        s = [ext[ch] for ch in lab]
        x = rng.uniform(-1, 1, s)
        return torch.from_numpy((x + 1j * rng.uniform(-1, 1, s) if np.issubdtype(dtype, np.complexfloating)
                                 else x).astype(dtype)).cuda()

    a, b, c, d = rand(la), rand(lb), rand(lc), rand(lc)
    v = [t1m.tensor(list(x.shape), x, t1m.row_major) for x in (a, b, c, d)]
    stream = torch.cuda.Stream()
    ctx = t1m.Context()
    ctx.set_stream(stream.cuda_stream)

    def calls():  # two products of the same operands, the second accumulating
        t1m.contract_raw(1.0, v[0], la, v[1], lb, 0.0, v[2], lc, t1m.FLAG_NO_TIMING, ctx)
        t1m.contract_raw(0.5, v[0], la, v[1], lb, 0.25, v[3], lc, t1m.FLAG_NO_TIMING, ctx)

    start = d.clone()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        calls()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        a.mul_(1.0)  # work of the caller's ahead of the products
        calls()
    for _ in range(3):
        a.copy_(rand(la))
        b.copy_(rand(lb))
        d.copy_(start)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        got = c.clone(), d.clone()
        d.copy_(start)
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            calls()
        torch.cuda.synchronize()
        assert torch.equal(got[0], c) and torch.equal(got[1], d)
    del graph
    ctx.close()
