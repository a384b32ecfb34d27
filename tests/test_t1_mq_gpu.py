"""MQ coding against the C oracle at the sizes where its launch changes (every block alone in a
warp, some alone, more blocks than a warp per scheduler takes, the last with one warp per scheduler
and the first with two (148 SMs), a batched launch's kernel), with
blocks of a few decisions to thousands and enough bytes that carries meet 0xFF bytes. Bytes and
whole numbers, so everything is compared exactly."""
import numpy as np
import pytest

import libgail_b200 as gb
from oracle.oracle import Oracle


@pytest.mark.gpu
@pytest.mark.parametrize("n,size,planes", [(1, 32, 12), (33, 32, 14), (700, 32, 9), (18900, 8, 12), (19000, 8, 12), (28416, 4, 9),
                                           (28417, 8, 9), (52000, 4, 9), (76000, 8, 9)])
def test_mq_matches_oracle(n, size, planes):
    rng = np.random.default_rng(n)
    top = 1 << (planes + 6)
    spread = np.exp2(rng.uniform(0, planes + 6, n))  # blocks from nearly empty to full
    m = np.zeros((n, 32, 32), np.uint32)
    m[:, :size, :size] = np.minimum(top - 1, rng.exponential(1.0, (n, size, size)) * spread[:, None, None])
    m |= ((rng.random((n, 32, 32)) < 0.5) & (m >= 64)).astype(np.uint32) << 31
    geom = np.stack([np.full(n, size), np.full(n, size), rng.integers(0, 4, n), np.full(n, 64)], 1).astype(np.int32)
    stride = 4096 if size == 32 else 512
    coeffs = m.reshape(n, 1024)
    want = Oracle().t1_encode_many(coeffs, geom, stride=stride)
    got = gb.t1_encode_blocks(coeffs, geom, data_stride=stride)
    assert np.array_equal(got[0][:, 1:], want[0][:, 1:])
    coded = np.arange(64) < want[0][:, 1:2]
    assert np.array_equal(np.where(coded, got[1], 0), np.where(coded, want[1], 0))
    assert got[3] == want[3]
