"""The launch queue: ops keep their order among each other and with writes and reads when there are more of them than the
ring holds, arguments and written bytes are taken at the call, wrong arguments are refused by the call that has them, and
the ops answer alike with the queue switched off."""
import ctypes as C
import threading

import numpy as np
import pytest

from gguf_trainer_b200 import _lib

pytestmark = pytest.mark.gpu
SCALE, ADD = 4, 0


@pytest.fixture(params=["1", "0"])
def gpu(request, monkeypatch):
    from gguf_trainer_b200.backend import requireGPU
    monkeypatch.setenv("GT_QUEUE", request.param)
    g = requireGPU("the queue suite", precision="fp32")
    yield g
    g.destroy()


def _buf(gpu, a):
    b = gpu.createStateBuffer(a.nbytes)
    gpu.writeStateBuffer(b, a)
    return b


def test_order_over_more_ops_than_the_ring_holds(gpu):
    lib, ctx, n = gpu.lib, gpu.ctx, 1000
    ones = np.ones(n, np.float32)
    x, one = _buf(gpu, np.zeros(n, np.float32)), _buf(gpu, ones)
    for i in range(3000):
        gpu._check(lib.gt_ew_fwd(ctx, ADD, n, x, one, 0.0, x))          # x += 1
        if i % 500 == 250:
            gpu._check(lib.gt_copy(ctx, one, x, 4 * n))                 # one = x, then back to ones by a write
            gpu._check(lib.gt_write(ctx, one, ones.ctypes.data, 4 * n))
        if i % 700 == 350:
            assert (gpu.readStateBuffer(x, n) == i + 1).all()
    assert (gpu.readStateBuffer(x, n) == 3000).all()
    gpu._check(lib.gt_zero(ctx, x, 4 * n))
    assert (gpu.readStateBuffer(x, n) == 0).all()


def test_arguments_are_taken_at_the_call(gpu):
    lib, ctx, n = gpu.lib, gpu.ctx, 64
    x = _buf(gpu, np.zeros(n, np.float32))
    outs = []
    host = np.empty(n, np.float32)
    for i in range(200):
        host[:] = i
        out = gpu.createStateBuffer(4 * n)
        gpu._check(lib.gt_write(ctx, x, host.ctypes.data, 4 * n))
        gpu._check(lib.gt_ew_fwd(ctx, SCALE, n, x, 0, 2.0, out))
        host[:] = -1
        outs.append(out)
    assert [gpu.readStateBuffer(o, n)[0] for o in outs] == [2.0 * i for i in range(200)]
    a, b = (_buf(gpu, np.arange(64, dtype=np.float32).reshape(8, 8) + k) for k in (0, 1))
    cs = [gpu.createStateBuffer(256) for _ in range(2)]
    m, p, q, acc = (C.c_int32 * 2)(8, 8), (C.c_uint64 * 2)(a, b), (C.c_uint64 * 2)(*cs), (C.c_int32 * 2)(0, 0)
    gpu._check(lib.gt_gemm_grouped(ctx, 0, 2, m, m, 8, p, p, q, acc))
    for v in (m, p, q, acc):
        C.memset(v, 0, C.sizeof(v))
    for k, c in enumerate(cs):
        A = np.arange(64.0).reshape(8, 8) + k
        assert np.array_equal(gpu.readStateBuffer(c, 64).reshape(8, 8), (A @ A.T).astype(np.float32))


def test_wrong_arguments_fail_at_their_call(gpu):
    lib, ctx, n = gpu.lib, gpu.ctx, 256
    x, y = _buf(gpu, np.ones(n, np.float32)), gpu.createStateBuffer(4 * n)
    for bad in (lambda: lib.gt_ew_fwd(ctx, ADD, n, x, 0, 0.0, y), lambda: lib.gt_ew_fwd(ctx, SCALE, n, x + 4, 0, 1.0, y),
                lambda: lib.gt_gemm(ctx, 0, 0, 0, 4, 4, x, x, y), lambda: lib.gt_rmsnorm_fwd(ctx, 1, 4096, x, x, 1e-5, y, y),
                lambda: lib.gt_rope_fwd(ctx, 1, 1, 3, 1e4, 0, x, y), lambda: lib.gt_attention_fwd(ctx, 4, 3, 2, 8, 0, x, x, x, y, y),
                lambda: lib.gt_glu_fwd(ctx, ADD, n, x, x, y), lambda: lib.gt_write(ctx, 0, None, 4)):
        gpu._check(lib.gt_ew_fwd(ctx, SCALE, n, x, 0, 3.0, y))
        assert bad() != 0 and lib.gt_last_error(ctx)
        with pytest.raises(_lib.GtError):
            gpu._check(bad())
        assert (gpu.readStateBuffer(y, n) == 3).all()
    with pytest.raises((C.ArgumentError, TypeError)):
        lib.gt_ew_fwd(ctx, ADD, n, "x", 0, 0.0, y)


def test_two_contexts_on_two_threads(gpu):
    from gguf_trainer_b200.backend import requireGPU
    other = requireGPU("the queue suite, second context", precision="fp32")
    got = {}

    def work(g, k):
        n = 512
        x, c = _buf(g, np.zeros(n, np.float32)), _buf(g, np.full(n, k, np.float32))
        for _ in range(1500):
            g._check(g.lib.gt_ew_fwd(g.ctx, ADD, n, x, c, 0.0, x))
        got[k] = g.readStateBuffer(x, n)

    threads = [threading.Thread(target=work, args=(g, k)) for g, k in ((gpu, 1), (other, 2))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    other.destroy()
    assert (got[1] == 1500).all() and (got[2] == 3000).all()
