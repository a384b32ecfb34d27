"""encoder_encode copies part of a frame's tables back before it knows their sizes: a frame that needs
more than that (or less) comes out as from an encoder of its own, whatever the frame before it was,
and takes the bus no longer. And
t1_encode_blocks keeps its device memory between calls: a small call after a large one, and calls
from several threads at once, give what each gives alone, and it is given back when it is asked
for or needed elsewhere."""
import threading

import numpy as np
import pytest
import torch

import libgail_b200 as gb
from libgail_b200 import plugin as P


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(1998, 1080), (64, 64)])
def test_sizes_of_the_frame_before(w, h):
    lay, fmt, col = P.LayoutHolder(w, h, 0), P.rgb48_format(w, h), P.color_passthrough()
    rng = np.random.default_rng(3)
    black, noise = np.zeros((h, w, 3), np.uint16), rng.integers(0, 65536, (h, w, 3)).astype(np.uint16)
    soft = (30000 + 300 * rng.standard_normal((h, w, 3))).astype(np.uint16)
    dev = P.Plugin().device(0)

    def alone(f):
        e = dev.encoder(lay, fmt, col)
        t = e.encode(f)[0]
        e.close()
        return t

    want = {k: alone(f) for k, f in (("black", black), ("noise", noise), ("soft", soft))}
    enc = dev.encoder(lay, fmt, col)
    for k in ("black", "noise", "soft", "noise", "black", "soft"):
        got = enc.encode({"black": black, "noise": noise, "soft": soft}[k])[0]
        for name in ("info", "pass_len", "pass_dist", "data"):
            assert np.array_equal(getattr(got, name), getattr(want[k], name)), (k, name)
    enc.close()
    dev.close()


@pytest.mark.gpu
def test_a_light_frame_after_a_heavy_one_copies_little():
    w, h = 3996, 2160
    enc = (dev := P.Plugin().device(0)).encoder(P.LayoutHolder(w, h, 1), P.rgb48_format(w, h), P.color_passthrough())
    noise, flat = np.random.default_rng(3).integers(0, 65536, (h, w, 3)).astype(np.uint16), np.zeros((h, w, 3), np.uint16)
    ms = {"noise": [], "flat": []}
    for _ in range(3):
        ms["noise"].append(enc.encode(noise)[1].download)  # 40 MB
        ms["flat"].append(enc.encode(flat)[1].download)  # next to nothing
    enc.close()
    dev.close()
    assert max(ms["flat"]) < 0.5 * min(ms["noise"]), ms


@pytest.mark.gpu
def test_blocks_memory_is_kept_safely():
    rng = np.random.default_rng(5)
    sets = []
    for n in (300, 3, 40, 1):
        c = np.minimum(16383, rng.exponential(900.0, (n, 1024))).astype(np.uint32)
        sets.append((c, np.tile(np.array([32, 32, 1, 64], np.int32), (n, 1))))
    want = [gb.t1_encode_blocks(*s, data_stride=4096) for s in sets]
    got = [None] * 8

    def call(i):
        for _ in range(3):
            got[i] = gb.t1_encode_blocks(*sets[i % len(sets)], data_stride=4096)

    threads = [threading.Thread(target=call, args=(i,)) for i in range(len(got))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i, g in enumerate(got):
        x = want[i % len(sets)]
        assert np.array_equal(g[0], x[0]) and g[3] == x[3]
        past = np.arange(64) >= x[0][:, 1:2]  # the tables whole: 0 past a block's passes
        for k in (1, 2):
            assert np.array_equal(g[k], x[k])
            assert not g[k][past].any()


@pytest.mark.gpu
def test_kept_memory_is_given_back():
    def call(n):
        c = np.full((n, 1024), 64, np.uint32)
        return gb.t1_encode_blocks(c, np.tile(np.array([32, 32, 0, 64], np.int32), (n, 1)), data_stride=4096)

    mb = 1 << 20
    gb.check(gb.lib().gb_t1_release_memory())
    call(1)  # whatever a first call loads
    gb.check(gb.lib().gb_t1_release_memory())
    free = torch.cuda.mem_get_info()[0]
    want = call(500)  # 59 MB, kept
    assert free - torch.cuda.mem_get_info()[0] >= 48 * mb
    gb.check(gb.lib().gb_t1_release_memory())
    assert free - torch.cuda.mem_get_info()[0] < 4 * mb
    call(500)
    hold = torch.empty(torch.cuda.mem_get_info()[0] - 90 * mb, dtype=torch.uint8, device="cuda")
    try:
        got = call(1000)  # 119 MB: only with the 59
    finally:
        del hold
        torch.cuda.empty_cache()
    assert got[3] == want[3] * 2
