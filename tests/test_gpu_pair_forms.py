"""The forms of the tensor-core product that CTA pairs carry (sums of products, groups, the gated unit, the rotation), at
sizes that leave remainders of their tiles; the tile is forced with `GT_GEMM_TILE`. References are f64 products of the same
f32 inputs."""
import ctypes as C

import numpy as np
import pytest

from gpu_harness import REL_L2_TC, rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from gguf_trainer_b200.backend import requireGPU
    g = requireGPU("the pair-form suite", precision="tf32")
    yield g
    g.destroy()


@pytest.fixture
def dev(gpu):
    held = []

    def put(a):
        b = gpu.createStateBuffer(a.nbytes)
        gpu.writeStateBuffer(b, np.ascontiguousarray(a, np.float32))
        held.append(b)
        return b
    yield put
    gpu.sync([])
    for b in held:
        gpu._check(gpu.lib.gt_free(gpu.ctx, b))


def _i32(*v):
    return (C.c_int32 * len(v))(*v)


def _ptr(v):
    return (C.c_uint64 * len(v))(*v)


def _read(gpu, b, shape):
    return gpu.readStateBuffer(b, int(np.prod(shape))).reshape(shape)


@pytest.mark.parametrize("tile", ["3,192", "3,256"])
@pytest.mark.parametrize("M,N,Ks,accum", [(513, 260, [576, 36, 100], 1), (129, 192, [40], 0), (2300, 576, [1536, 1536], 0)])
def test_sum_of_products(gpu, dev, monkeypatch, tile, M, N, Ks, accum):
    monkeypatch.setenv("GT_GEMM_TILE", tile)
    rng = np.random.default_rng(M)
    A = [rng.standard_normal((M, k), dtype=np.float32) for k in Ks]
    B = [rng.standard_normal((k, N), dtype=np.float32) for k in Ks]
    c0 = rng.standard_normal((M, N), dtype=np.float32)
    c = dev(c0)
    gpu._check(gpu.lib.gt_gemm_multi(gpu.ctx, 1, accum, M, N, len(Ks), _i32(*Ks), _ptr([dev(a) for a in A]), _ptr([dev(b) for b in B]), c))
    want = sum(a.astype(np.float64) @ b for a, b in zip(A, B)) + (c0 if accum else 0.0)
    assert rel_l2(_read(gpu, c, (M, N)), want) <= REL_L2_TC


@pytest.mark.parametrize("tile", ["2,256", "3,192", "3,256"])
@pytest.mark.parametrize("kind,K,shapes", [(2, 1030, [(576, 192), (64, 260), (16, 1024)]), (0, 96, [(700, 576), (700, 192), (700, 32)]),
                                           (1, 2080, [(300, 64), (130, 516)])])
def test_groups(gpu, dev, monkeypatch, tile, kind, K, shapes):
    K -= K % 4
    monkeypatch.setenv("GT_GEMM_TILE", tile)
    rng = np.random.default_rng(K)
    A = [rng.standard_normal((m, K), dtype=np.float32) for m, _ in shapes]
    B = [rng.standard_normal((n, K), dtype=np.float32) for _, n in shapes]
    c0 = [rng.standard_normal(s, dtype=np.float32) for s in shapes]
    cs = [dev(c) for c in c0]
    acc = [g % 2 for g in range(len(shapes))]
    gpu._check(gpu.lib.gt_gemm_grouped(gpu.ctx, kind, len(shapes), _i32(*[m for m, _ in shapes]), _i32(*[n for _, n in shapes]), K,
                                       _ptr([dev(a.T if kind == 2 else a) for a in A]), _ptr([dev(b if kind == 0 else b.T) for b in B]),
                                       _ptr(cs), _i32(*acc)))
    for a, b, c, z, ac, s in zip(A, B, cs, c0, acc, shapes):
        assert rel_l2(_read(gpu, c, s), a.astype(np.float64) @ b.T + (z if ac else 0.0)) <= REL_L2_TC


@pytest.mark.parametrize("tile", ["3,192", "3,256"])
@pytest.mark.parametrize("rows,T", [(514, 257), (70, 70)])
def test_rotated_group(gpu, dev, monkeypatch, tile, rows, T):
    monkeypatch.setenv("GT_GEMM_TILE", tile)
    rng = np.random.default_rng(rows)
    h, outs = 100, (320, 128, 64)
    x = rng.standard_normal((rows, h), dtype=np.float32)
    W = [rng.standard_normal((o, h), dtype=np.float32) for o in outs]
    ys = [dev(np.zeros((rows, o), np.float32)) for o in outs]
    gpu.setBatch(rows // T, T)
    try:
        gpu._check(gpu.lib.gt_linear_rope_grouped(gpu.ctx, 3, rows, h, dev(x), _i32(*outs), _ptr([dev(w) for w in W]), _ptr(ys), _i32(5, 2, 0), 64, 1e4, 0))
        got = [_read(gpu, y, (rows, o)) for y, o in zip(ys, outs)]
    finally:
        gpu.setBatch(0, 0)
    ang = (np.arange(rows) % T)[:, None] * 1e4 ** (-np.arange(32) / 32.0)
    for y, w, rotated in zip(got, W, (True, True, False)):
        want = x.astype(np.float64) @ w.T
        if rotated:
            v = want.reshape(rows, -1, 64)
            c, s = np.cos(ang)[:, None], np.sin(ang)[:, None]
            want = np.concatenate([v[..., :32] * c - v[..., 32:] * s, v[..., :32] * s + v[..., 32:] * c], -1).reshape(rows, -1)
        assert rel_l2(y, want) <= REL_L2_TC


@pytest.mark.parametrize("op", [2, 3])
@pytest.mark.parametrize("rows,h,ffn", [(300, 100, 420), (129, 576, 128)])
def test_gated_unit(gpu, dev, monkeypatch, op, rows, h, ffn):
    monkeypatch.setenv("GT_GEMM_TILE", "3,256")
    rng = np.random.default_rng(ffn)
    x, wg, wu = (rng.standard_normal(s, dtype=np.float32) for s in ((rows, h), (ffn, h), (ffn, h)))
    outs = [dev(np.zeros((rows, ffn), np.float32)) for _ in range(3)]
    gpu._check(gpu.lib.gt_glu_linear_fwd(gpu.ctx, op, rows, ffn, h, dev(x), dev(wg), dev(wu), *outs))
    g, u = x.astype(np.float64) @ wg.T, x.astype(np.float64) @ wu.T
    act = g / (1 + np.exp(-g)) if op == 2 else 0.5 * g * (1 + np.tanh(0.7978845608028654 * (g + 0.044715 * g ** 3)))
    for b, want in zip(outs, (g, u, act * u)):
        assert rel_l2(_read(gpu, b, (rows, ffn)), want) <= 2 * REL_L2_TC
