"""gt_read and gt_read_many around the sizes of their staging blocks: single bytes, arrays that share a block, arrays that
end on, before and after a block's edge, more bytes than the staging ring holds, zero-length entries."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

K = 1024


@pytest.fixture(scope="module")
def gpu():
    from gguf_trainer_b200.backend import requireGPU
    g = requireGPU("the read suite")
    yield g
    g.destroy()


@pytest.mark.parametrize("sizes", [[1], [64 * K], [64 * K + 1], [128 * K - 1, 1, 128 * K + 1], [512 * K, 512 * K, 3], [7] * 300, [0, 5, 0, 4096, 0],
                                   [40 * 1024 * K + 12345], [3 * 1024 * K + 7] * 9 + [64, 0, 1]])
def test_sizes(gpu, sizes):
    src = [np.random.default_rng(i).integers(0, 256, n, dtype=np.uint8) for i, n in enumerate(sizes)]
    dev = [gpu.createStateBuffer(max(n, 4)) for n in sizes]
    for d, s in zip(dev, src):
        gpu._write(d, s) if s.size else None
    for _ in range(2):
        out = [np.zeros(n, np.uint8) for n in sizes]
        n = len(sizes)
        gpu._check(gpu.lib.gt_read_many(gpu.ctx, n, (C.c_uint64 * n)(*dev), (C.c_void_p * n)(*[o.ctypes.data for o in out]), (C.c_uint64 * n)(*sizes)))
        assert all(np.array_equal(a, b) for a, b in zip(out, src))
    one = np.zeros(sizes[-1], np.uint8)
    gpu._read(dev[-1], one)
    assert np.array_equal(one, src[-1])
    for d in dev:
        gpu._check(gpu.lib.gt_free(gpu.ctx, d))
