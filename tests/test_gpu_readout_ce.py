"""The chunked readout loss with its statistics and its gradient taken in the product's epilogue, at the edges of its
tiles: rows and columns that leave remainders, spans whose targets lie inside and outside, ignored rows, the fused form
and the two-pass form (`GT_GEMM_TILE`). References are f64 products of the same f32 inputs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from gguf_trainer_b200.backend import requireGPU
    g = requireGPU("the chunked readout suite", precision="tf32")
    yield g
    g.destroy()


@pytest.mark.parametrize("tile", ["3,256", "1,192"])
@pytest.mark.parametrize("rows,h,spans", [(1000, 96, [1920, 1920, 700]), (257, 40, [16384, 4]), (16, 16, [30720, 30001])])
def test_readout_ce(gpu, monkeypatch, tile, rows, h, spans):
    monkeypatch.setenv("GT_GEMM_TILE", tile)
    rng = np.random.default_rng(rows)
    V = sum(spans)
    x, w = rng.standard_normal((rows, h), dtype=np.float32), rng.standard_normal((V, h), dtype=np.float32)
    tg = rng.integers(0, V, rows).astype(np.uint32)
    tg[::3] = 0xFFFFFFFF
    tg[1], tg[-1] = 0, V - 1
    z = x.astype(np.float64) @ w.astype(np.float64).T
    kept = tg != 0xFFFFFFFF
    lse = np.log(np.exp(z - z.max(1, keepdims=True)).sum(1)) + z.max(1)
    inv = 1.0 / kept.sum()
    want = np.exp(z - lse[:, None])
    want[np.arange(rows)[kept], tg[kept]] -= 1
    want *= kept[:, None] * inv

    def dev(a):
        b = gpu.createStateBuffer(a.nbytes)
        gpu.writeStateBuffer(b, np.ascontiguousarray(a).view(np.float32))
        return b

    dx, dw, dt, di, dl = dev(x), dev(w), dev(tg), dev(np.array([inv], np.float32)), dev(np.ones(1, np.float32))
    run, chunk = gpu.createStateBuffer(rows * 12), gpu.createStateBuffer(rows * max(spans) * 4)
    v0 = 0
    for i, n in enumerate(spans):
        gpu._check(gpu.lib.gt_readout_ce_stats(gpu.ctx, rows, n, h, v0, 1 if i == 0 else 0, dx, dw + v0 * h * 4, chunk, dt, run))
        v0 += n
    m, s, t = gpu.readStateBuffer(run, rows * 3).reshape(rows, 3).astype(np.float64).T
    scale = np.abs(z).max()
    assert np.abs(np.log(s) + m - lse).max() <= 2e-3 * scale
    assert np.abs(t[kept] - z[np.arange(rows)[kept], tg[kept]]).max() <= 2e-3 * scale
    assert (t[~kept] == 0).all()
    v0 = 0
    for n in spans:
        gpu._check(gpu.lib.gt_readout_ce_grad(gpu.ctx, rows, n, h, v0, dx, dw + v0 * h * 4, chunk, dt, run, di, dl))
        got = gpu.readStateBuffer(chunk, rows * n).reshape(rows, n)
        assert (got[~kept] == 0).all()
        assert np.linalg.norm(got - want[:, v0:v0 + n]) <= 5e-3 * np.linalg.norm(want)
        v0 += n
    # the whole vocabulary at once, logits kept
    V4 = V - V % 4
    t4 = np.where(tg < V4, tg, 0xFFFFFFFF).astype(np.uint32)
    k4 = t4 != 0xFFFFFFFF
    lg, st, ls, ik, d4 = (gpu.createStateBuffer(n) for n in (rows * V4 * 4, rows * 16, 8, 4, rows * 4))
    gpu.writeStateBuffer(d4, t4.view(np.float32))
    gpu._check(gpu.lib.gt_readout_ce_fwd(gpu.ctx, rows, V4, h, dx, dw, lg, d4, st, ls, ik))
    assert np.linalg.norm(gpu.readStateBuffer(lg, rows * V4).reshape(rows, V4) - z[:, :V4]) <= 2e-3 * np.linalg.norm(z)
    m4 = z[:, :V4].max(1)
    lse4 = np.log(np.exp(z[:, :V4] - m4[:, None]).sum(1)) + m4
    S = gpu.readStateBuffer(st, rows * 4).reshape(rows, 4).astype(np.float64)
    nll = np.where(k4, lse4 - z[np.arange(rows), np.where(k4, t4, 0)], 0.0)
    assert np.abs(S[:, 0] - np.log(S[:, 1]) - lse4).max() <= 2e-3 * scale and np.abs(S[:, 2] - nll).max() <= 4e-3 * scale
    assert abs(gpu.readStateBuffer(ls, 1)[0] - nll.sum() / k4.sum()) <= 2e-3 * scale
    gpu.sync([])
    for b in (dx, dw, dt, di, dl, run, chunk, lg, st, ls, ik, d4):
        gpu._check(gpu.lib.gt_free(gpu.ctx, b))
