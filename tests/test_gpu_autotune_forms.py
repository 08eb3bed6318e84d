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
