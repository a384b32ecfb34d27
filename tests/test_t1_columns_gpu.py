"""Context modelling on whole columns against the C oracle, at the sizes and contents where the
row masks can go wrong: partial stripes and columns, every orientation, one to many planes,
pass limits, empty and full blocks, long significance chains, runs. Everything is whole numbers,
so everything is compared exactly."""
import numpy as np
import pytest

import libgail_b200 as gb
from oracle.oracle import Oracle

SIZES = [(1, 1), (1, 32), (32, 1), (2, 3), (3, 4), (4, 5), (5, 8), (31, 31), (32, 31), (31, 32), (32, 32), (17, 29)]


def _contents(rng, planes):
    """Magnitude words (6 fraction bits) of 32 x 32 blocks with at most `planes` bit-planes."""
    top = 1 << (planes + 6)
    flat = rng.integers(0, top, (32, 32))
    yield flat
    yield np.zeros((32, 32), np.int64)
    yield np.full((32, 32), top - 1)
    yield np.where(rng.random((32, 32)) < 0.02, flat, 0)                 # mostly runs
    yield np.minimum(top - 1, rng.exponential(top / 24, (32, 32)).astype(np.int64))
    yield np.where(np.add.outer(np.arange(32), np.arange(32)) % 7 == 0, top - 1, 64)  # diagonal chains
    row, col = np.mgrid[:32, :32]
    yield np.where(row % 4 == 3, top - 1, top // 2)                      # stripes' last rows first
    yield np.where(col == 31, top - 1, 70)                               # chains towards the left


@pytest.mark.gpu
@pytest.mark.parametrize("planes", [1, 2, 9, 22])
@pytest.mark.parametrize("max_passes", [64, 5])
def test_columns_match_oracle(planes, max_passes):
    rng = np.random.default_rng(planes * 100 + max_passes)
    coeffs, geom = [], []
    for w, h in SIZES:
        for orient in range(4):
            for m in _contents(rng, planes):
                sign = (rng.random((32, 32)) < 0.5) & (m >= 64)
                coeffs.append((m.astype(np.uint32) | (sign.astype(np.uint32) << 31)).ravel())
                geom.append((w, h, orient, max_passes))
    coeffs, geom = np.array(coeffs), np.array(geom, np.int32)
    clean = coeffs.reshape(-1, 32, 32).copy()  # the library takes words outside w x h as 0; so must the oracle
    for i, (w, h, _, _) in enumerate(geom):
        clean[i, h:, :] = 0
        clean[i, :, w:] = 0
    want = Oracle().t1_encode_many(clean.reshape(-1, 1024), geom)
    got = gb.t1_encode_blocks(coeffs, geom)
    assert np.array_equal(got[0][:, 1:], want[0][:, 1:])  # passes, decisions, bytes
    coded = np.arange(64) < want[0][:, 1:2]
    assert np.array_equal(np.where(coded, got[1], 0), np.where(coded, want[1], 0))
    assert np.array_equal(np.where(coded, got[2], 0), np.where(coded, want[2], 0))
    assert got[3] == want[3]
