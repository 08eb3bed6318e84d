"""The tuner measures the streamed form too: a permuted contraction to a small
matrix over a long bundle, whose streamed form takes two thirds of the others'
time, is tuned to it and keeps it from the cache (gpu)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_tuner_streams(ctx, torch_cuda, tmp_path, monkeypatch):
    import t1m_gb300 as t1m
    torch = torch_cuda
    monkeypatch.setenv("T1M_TUNE_CACHE", str(tmp_path / "tune.txt"))
    ext = dict(a=24, b=32, c=96, d=48, e=64)
    rng = np.random.default_rng(52)

    def rand(labels):
        s = [ext[ch] for ch in labels]
        return (rng.uniform(-1, 1, s) + 1j * rng.uniform(-1, 1, s)).astype(np.complex64)

    A, B = rand("abcd"), rand("dbea")
    ga, gb = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    v = lambda z: t1m.tensor(list(z.shape), z, t1m.row_major)  # noqa: E731
    ref = np.einsum("abcd,dbea->ec", A.astype(np.complex128), B.astype(np.complex128))
    reps = []
    ctx.set_autotune(True)
    try:
        for _ in range(2):  # tuned, then from the cache
            gc = torch.zeros((64, 96), dtype=torch.complex64, device="cuda")
            torch.cuda.synchronize()
            reps.append(t1m.contract_scaled(1.0, v(ga), "abcd", v(gb), "dbea", 0.0, v(gc), "ec",
                                            ctx=ctx))
            torch.cuda.synchronize()
            assert np.abs(gc.cpu().numpy() - ref).max() <= 1e-6 * np.abs(ref).max()
    finally:
        ctx.set_autotune(False)
    lines = (tmp_path / "tune.txt").read_text().splitlines()
    codes = [int(x.split()[1]) for x in lines[1:] if x.startswith("s:2:")]
    assert codes == [900], lines
    assert reps[0].split_k == reps[1].split_k > 76 and reps[1].kernels == 2


def test_group_tuner_tells_pieces_apart(built_lib, torch_cuda, tmp_path, monkeypatch):
    """Items over operand pieces and items that split in the kernel (a capped
    workspace) are tuned and cached apart: what is fastest over pieces need not
    be without them."""
    import t1m_gb300 as t1m
    torch = torch_cuda
    monkeypatch.setenv("T1M_TUNE_CACHE", str(tmp_path / "tune.txt"))
    rng = np.random.default_rng(53)

    def rand(*s):
        x = (rng.uniform(-1, 1, s) + 1j * rng.uniform(-1, 1, s)).astype(np.complex64)
        return torch.from_numpy(x).cuda()

    v = lambda z: t1m.tensor(list(z.shape), z, t1m.row_major)  # noqa: E731
    shapes = [(96, 80, 200), (300, 3, 400)]
    ops = [(rand(m, k), rand(k, n)) for m, n, k in shapes]
    for limit in (-1, 0):
        ctx = t1m.Context()
        ctx.set_workspace_limit(limit)
        outs = [torch.zeros((m, n), dtype=torch.complex64, device="cuda") for m, n, _ in shapes]
        torch.cuda.synchronize()
        g = t1m.Group([(1.0, v(a), "mk", v(b), "kn", 0.0, v(c), "mn", -1)
                       for (a, b), c in zip(ops, outs)], ctx=ctx, autotune=True)
        g.launch()
        torch.cuda.synchronize()
        for (a, b), c in zip(ops, outs):
            ref = a.to(torch.complex128) @ b.to(torch.complex128)
            assert (c - ref).abs().max() <= 1e-6 * ref.abs().max()
        g.close()
        ctx.close()
    keys = [x.split()[0] for x in (tmp_path / "tune.txt").read_text().splitlines()[1:]]
    assert sorted(keys) == ["2:6,6,7", "2:8,1,8", "p2:6,6,7", "p2:8,1,8"]
