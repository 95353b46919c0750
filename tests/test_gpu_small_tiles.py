"""The kernels that carry small work, at the sizes where their tiles can go wrong: the one-tile-per-CTA tensor-core
product (`GT_GEMM_TILE=0,bn` forces it), the strict-f32 product's two tiles and its cluster reduction, and the strict-f32
attention's row and column tiles, head padding, windows and shared groups. References are f64 products of the same f32
inputs and the CPU oracle."""
import ctypes as C

import numpy as np
import pytest

from gpu_harness import REL_L2_FP32, REL_L2_TC, op_case, rand_tensor, rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["tf32", "fp32"])
def gpu(request):
    from gguf_trainer_b200.backend import requireGPU
    g = requireGPU("the small-tile suite", precision=request.param)
    yield g
    g.destroy()


def _dev(gpu, a):
    b = gpu.createStateBuffer(a.nbytes)
    gpu.writeStateBuffer(b, np.ascontiguousarray(a))
    return b


def _product(gpu, kind, M, N, K, accum, seed):
    rng = np.random.default_rng(seed)
    A, B, C0 = (rng.standard_normal(s, dtype=np.float32) for s in ((M, K), (N, K), (M, N)))
    bufs = [_dev(gpu, A.T if kind == "TN" else A), _dev(gpu, B if kind == "NT" else B.T), _dev(gpu, C0)]
    gpu._gemm(kind, accum, M, N, K, *bufs)
    got = gpu.readStateBuffer(bufs[2], M * N).reshape(M, N)
    gpu.sync([])
    for b in bufs:
        gpu._check(gpu.lib.gt_free(gpu.ctx, b))
    return rel_l2(got, A.astype(np.float64) @ B.astype(np.float64).T + (C0 if accum else 0.0))


@pytest.mark.parametrize("bn", ["32", "64", "128"])
@pytest.mark.parametrize("kind,M,N,K,accum", [("NT", 37, 576, 576, 0), ("NT", 129, 49, 96, 1), ("NN", 256, 132, 1536, 1),
                                              ("TN", 576, 192, 260, 0), ("TN", 16, 1024, 2048, 1), ("NT", 16, 16, 16, 0),
                                              ("NT", 40, 4096, 36, 0)])
def test_product_one_tile_per_cta(gpu, monkeypatch, bn, kind, M, N, K, accum):
    monkeypatch.setenv("GT_GEMM_TILE", "0," + bn)
    r = _product(gpu, kind, M, N, K, accum, M + N + K)
    assert r <= (REL_L2_TC if gpu.precision == "tf32" else REL_L2_FP32), r


@pytest.mark.parametrize("kind,M,N,K,accum", [("NT", 1, 1, 1, 0), ("NT", 65, 63, 33, 1), ("NN", 63, 129, 31, 0), ("TN", 64, 64, 2100, 1),
                                              ("TN", 70, 6, 515, 0), ("NT", 1300, 1200, 20, 0), ("NN", 5, 7, 4100, 1)])
def test_product_ragged(gpu, kind, M, N, K, accum):
    r = _product(gpu, kind, M, N, K, accum, 3 * M + N + K)
    assert r <= (REL_L2_TC if gpu.precision == "tf32" else REL_L2_FP32), r


@pytest.mark.parametrize("tile", ["", "0,64", "0,128"])
@pytest.mark.parametrize("rows", [40, 130])
def test_grouped_rotated_and_gated(gpu, monkeypatch, tile, rows):
    """q, k, v of one input with q and k rotated, and gate, up and the gated unit, as the step launches them."""
    if tile:
        monkeypatch.setenv("GT_GEMM_TILE", tile)
    tol = REL_L2_TC if gpu.precision == "tf32" else REL_L2_FP32
    rng = np.random.default_rng(rows)
    K, Ns, heads = 192, (128, 64, 64), (2, 1, 0)
    x = rng.standard_normal((rows, K), dtype=np.float32)
    ws = [rng.standard_normal((n, K), dtype=np.float32) for n in Ns]
    dx, dw, dy = _dev(gpu, x), [_dev(gpu, w) for w in ws], [gpu.createStateBuffer(rows * n * 4) for n in Ns]
    gpu._check(gpu.lib.gt_linear_rope_grouped(gpu.ctx, 3, rows, K, dx, (C.c_int32 * 3)(*Ns), (C.c_uint64 * 3)(*dw), (C.c_uint64 * 3)(*dy),
                                              (C.c_int32 * 3)(*heads), 64, 10_000.0, 0))
    ang = np.arange(rows)[:, None] * 10_000.0 ** (-np.arange(32) * 2.0 / 64)
    for n, h, w, d in zip(Ns, heads, ws, dy):
        want = (x.astype(np.float64) @ w.astype(np.float64).T)
        if h:
            y = want.reshape(rows, h, 2, 32)
            c, s = np.cos(ang)[:, None], np.sin(ang)[:, None]
            want = np.stack([y[:, :, 0] * c - y[:, :, 1] * s, y[:, :, 0] * s + y[:, :, 1] * c], 2).reshape(rows, n)
        assert rel_l2(gpu.readStateBuffer(d, rows * n), want) <= tol
    ffn = 100
    wg, wu = (rng.standard_normal((ffn, K), dtype=np.float32) / 14 for _ in range(2))
    outs = [gpu.createStateBuffer(rows * ffn * 4) for _ in range(3)]
    bufs = [_dev(gpu, wg), _dev(gpu, wu)]
    gpu._check(gpu.lib.gt_glu_linear_fwd(gpu.ctx, 2, rows, ffn, K, dx, *bufs, *outs))
    g, u = x.astype(np.float64) @ wg.T, x.astype(np.float64) @ wu.T
    for b, want in zip(outs, (g, u, g / (1 + np.exp(-g)) * u)):
        assert rel_l2(gpu.readStateBuffer(b, rows * ffn), want) <= tol
    gpu.sync([])
    for b in [dx] + dw + dy + outs + bufs:
        gpu._check(gpu.lib.gt_free(gpu.ctx, b))


@pytest.mark.parametrize("T,Hq,Hkv,hd,window", [(1, 2, 1, 8, 0), (33, 3, 1, 6, 0), (65, 6, 2, 64, 0), (130, 8, 1, 24, 40), (64, 9, 3, 128, 0),
                                                (97, 4, 1, 256, 33), (40, 10, 1, 100, 0)])
def test_strict_f32_attention_tiles(gpu, oracle, T, Hq, Hkv, hd, window):
    if gpu.precision != "fp32":
        pytest.skip("the f32 kernels")
    from gguf_trainer_b200 import autograd as ag
    rng = oracle.Mulberry32(T + hd)
    q, k, v = rand_tensor(rng, [T, Hq * hd]), rand_tensor(rng, [T, Hkv * hd]), rand_tensor(rng, [T, Hkv * hd])

    def ref(r):
        out, grads = _attention_f64(q, k, v, T, Hq, Hkv, hd, window, r)
        return [out], grads

    def ref1(r):
        o, g = ref(r)
        return o[0], g

    op_case(gpu, oracle, f"attention {T} {Hq}/{Hkv}x{hd} w{window}", [q, k, v], lambda: ag.attention(q, k, v, T, Hq, Hkv, hd, window), ref1)


def _attention_f64(q, k, v, T, Hq, Hkv, hd, window, up):
    Q, K, V, G = (t.astype(np.float64).reshape(T, -1, hd) for t in (q.data, k.data, v.data, up))
    gq, gk, gv, out = np.zeros_like(Q), np.zeros_like(K), np.zeros_like(V), np.zeros_like(Q)
    i, j = np.arange(T)[:, None], np.arange(T)[None]
    keep = (j <= i) & ((window == 0) | (j > i - window))
    for h in range(Hq):
        n = h // (Hq // Hkv)
        s = np.where(keep, Q[:, h] @ K[:, n].T / np.sqrt(hd), -np.inf)
        p = np.exp(s - s.max(1, keepdims=True))
        p /= p.sum(1, keepdims=True)
        out[:, h] = p @ V[:, n]
        dp = G[:, h] @ V[:, n].T
        ds = p * (dp - (dp * p).sum(1, keepdims=True)) / np.sqrt(hd)
        gv[:, n] += p.T @ G[:, h]
        gq[:, h] = ds @ K[:, n]
        gk[:, n] += ds.T @ Q[:, h]
    return out.reshape(-1), [gq.reshape(-1), gk.reshape(-1), gv.reshape(-1)]


@pytest.mark.parametrize("d", [64, 576, 1024])
@pytest.mark.parametrize("rows", [1, 16, 17, 127, 128, 129, 513])
def test_norm_backward_few_rows(gpu, d, rows):
    """dw over one CTA, one cluster (up to 128 rows), and beyond it; overwriting and adding."""
    rng = np.random.default_rng(rows + d)
    x, g, gadd = (rng.standard_normal((rows, d), dtype=np.float32) for _ in range(3))
    w, gw0 = rng.standard_normal(d, dtype=np.float32), rng.standard_normal(d, dtype=np.float32)
    X = x.astype(np.float64)
    r = 1.0 / np.sqrt((X * X).mean(1) + 1e-5)
    rinv = r.astype(np.float32)
    want_x = w * r[:, None] * g - X * (r ** 3 * (g * w * X).sum(1) / d)[:, None]
    want_w = (g * X * r[:, None]).sum(0)
    bufs = dx, dw, dr, dg, da, do, dgw = [_dev(gpu, a) for a in (x, w, rinv, g, gadd, x, gw0)]
    for acc in (1, 0):
        gpu._check(gpu.lib.gt_rmsnorm_bwd_add(gpu.ctx, rows, d, dx, dw, dr, dg, da, do, dgw, acc))
        assert rel_l2(gpu.readStateBuffer(dgw, d), want_w + (gw0 if acc else 0.0)) <= REL_L2_FP32
        assert rel_l2(gpu.readStateBuffer(do, rows * d), want_x + gadd) <= REL_L2_FP32
    gpu.sync([])
    for b in bufs:
        gpu._check(gpu.lib.gt_free(gpu.ctx, b))
