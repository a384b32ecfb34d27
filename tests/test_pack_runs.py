"""gb_t1_encode_blocks brings codewords back in runs whose packed bytes stay below a limit, as
packed offsets are 32 bits: the runs themselves without a GPU, a call of several runs with one."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import libgail_b200 as gb
from oracle.oracle import Oracle

CSRC = os.path.join(os.path.dirname(os.path.abspath(gb.__file__)), "csrc")


@pytest.fixture(scope="module")
def packed_run(tmp_path_factory):
    d = tmp_path_factory.mktemp("pack_runs")
    (d / "t.cpp").write_text('#include "pack_runs.h"\nextern "C" uint32_t run(const uint32_t* i, uint32_t f, uint32_t n, '
                             'uint64_t l, uint64_t* b) { return gb::packedRun(i, f, n, l, *b); }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "t.cpp"), "-o", str(d / "t.so")], check=True)
    fn = C.CDLL(str(d / "t.so")).run
    fn.restype = C.c_uint32
    fn.argtypes = [C.c_void_p, C.c_uint32, C.c_uint32, C.c_uint64, C.c_void_p]
    return fn


@pytest.mark.parametrize("lens,limit", [
    ([0] * 5, 64), ([1, 2, 3, 4, 5], 8), ([100, 1, 1], 8), ([8, 8, 8], 16), ([7, 0, 0, 9, 0], 8),
    ([0xFFFFFFFF, 1, 0xFFFFFFF0, 5], 1 << 33),             # whole words and sums past 32 bits
    ([3000] * 2_000_000, 64 << 20), ([3000] * 2_000_000, (1 << 32) - 4),  # 6 GB together
])
def test_runs_cover_the_blocks_within_the_limit(packed_run, lens, limit):
    info = np.zeros((len(lens), 4), np.uint32)
    info[:, 3] = lens
    words = (np.array(lens, np.uint64) + np.uint64(3)) & ~np.uint64(3)
    first = 0
    while first < len(lens):
        b = C.c_uint64()
        end = packed_run(info.ctypes.data, first, len(lens), limit, C.byref(b))
        assert first < end <= len(lens)
        assert b.value == int(words[first:end].sum())
        assert b.value <= limit or end == first + 1
        assert end == len(lens) or b.value + int(words[end]) > limit  # as long as it can be
        first = end


@pytest.mark.gpu
def test_several_runs_match_oracle():
    rng = np.random.default_rng(11)
    m = rng.integers(0, 1 << 28, (96, 1024), dtype=np.uint32)
    m[::7] = 0
    m[1::7] = np.minimum(m[1::7], 1 << 20)
    geom = np.stack([np.full(96, 32), np.full(96, 32), rng.integers(0, 4, 96), np.full(96, 64)], 1).astype(np.int32)
    want = Oracle().t1_encode_many(m, geom, stride=8192)
    reps = 64 * (1 << 20) // sum(len(c) for c in want[3]) + 130  # past one run of 64 MB
    got = gb.t1_encode_blocks(np.tile(m, (reps, 1)), np.tile(geom, (reps, 1)), data_stride=8192)
    assert sum(map(len, got[3])) > 64 << 20
    assert np.array_equal(got[0][:, 1:], np.tile(want[0][:, 1:], (reps, 1)))
    assert all(g == want[3][i % 96] for i, g in enumerate(got[3]))
