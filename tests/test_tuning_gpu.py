"""Tuning changes launch shapes and work order, never results: Tier-1 frames and decoded
pictures are bit-identical under extreme tunings, and so are the frames of batched launches, where
the MQ coding's knobs act (above 128 blocks per scheduler)."""
import numpy as np
import pytest
import torch

from libgail_b200 import autotune as AT
from libgail_b200 import codestream as CS
from libgail_b200 import plugin as P
from libgail_b200 import synth
from libgail_b200.engine import Engine
from oracle.oracle import Oracle


@pytest.mark.gpu
def test_tuning_does_not_change_results():
    W, H = 1998, 1080
    dev = P.Plugin().device(0)
    lay = P.LayoutHolder(W, H, 0)
    frame = synth.xyz12_to_rgb48(synth.xyz12_planes(W, H, seed=77))
    try:
        enc = dev.encoder(lay, P.rgb48_format(W, H), P.color_passthrough())
        ref = enc.encode(frame)[0]
        cs = CS.rate_and_build(lay, ref, 24.0)[0]
        blocks = CS.parse(cs)[1].view(P.CBLK_CODE_DTYPE)
        dec = dev.decoder(lay)
        pic = dec.decode(cs, blocks)[0]
        for t in ({"soloDecisions": 256, "cmCtasPerSm": 1, "mqCtasPerSm": 1, "decCtasPerSm": 1},
                  {"soloDecisions": 1 << 30, "cmCtasPerSm": 64, "mqCtasPerSm": 64, "decCtasPerSm": 64}):
            AT.set_tuning(0, t)
            got = enc.encode(frame)[0]
            assert np.array_equal(got.info, ref.info) and np.array_equal(got.data, ref.data)
            assert np.array_equal(got.pass_len, ref.pass_len) and np.array_equal(got.pass_dist, ref.pass_dist)
            assert np.array_equal(dec.decode(cs, blocks)[0], pic)
        dec.close()
        enc.close()
    finally:
        AT.set_tuning(0, None)
        dev.close()


@pytest.mark.gpu
@pytest.mark.parametrize("tuning", [{}, {"soloDecisions": 16384, "cmCtasPerSm": 1, "mqCtasPerSm": 1},
                                    {"soloDecisions": 1 << 30, "cmCtasPerSm": 64, "mqCtasPerSm": 64}])
def test_batched_launches_under_extreme_tuning(tuning):
    """4K frames in batches of three and more (77,958 blocks; two launches order them, the wide
    MQ kernel codes them) against the frames encoded alone, one of them against the oracle too."""
    W, H = 3996, 2160
    dev = P.Plugin().device(0)
    lay, fmt, col = P.LayoutHolder(W, H, 1), P.rgb48_format(W, H), P.color_passthrough()
    assert 3 * lay.num_cblks > 128 * 4 * torch.cuda.get_device_properties(0).multi_processor_count
    frames = [synth.xyz12_to_rgb48(synth.xyz12_planes(W, H, seed=70 + i)) for i in range(2)]
    enc = dev.encoder(lay, fmt, col)
    want = [enc.encode(frames[1])[0]]
    t1, _, taps = enc.encode(frames[0], debug=True)
    want.insert(0, t1)
    some = np.arange(0, lay.num_cblks, 37)
    geom = np.array([(min(32, b.w - 32 * (k % b.ncbx)), min(32, b.h - 32 * (k // b.ncbx)), b.orient, 64)
                     for b in lay.bands for k in range(b.ncbx * b.ncby)], np.int32)
    o = Oracle().t1_encode_many(taps["coeffs"].reshape(-1, 1024)[some], geom[some], stride=8192)
    for k, i in enumerate(some):
        assert t1.block(i)[2] == o[3][k]
        assert np.array_equal(t1.block(i)[3], o[1][k, :t1.info[i, 1]])
    enc.close()
    on_gpu = [torch.from_numpy(f.view(np.int16)).cuda() for f in frames]
    eng = Engine(0, 0, max_batch=8)
    try:
        AT.set_tuning(1, tuning)
        cls, _ = eng.add_encoder(lay, fmt, col)
        eng.reserve(cls, 16)
        eng.set_policy(8, 100, 1000.0)
        wide = False  # some batch of a burst had three frames or more
        for _ in range(10):
            before = eng.stats()
            which = {eng.submit(cls, on_gpu[i % 2]): i % 2 for i in range(16)}
            for _ in range(16):
                rid, got, _, st = eng.wait(60000)
                assert rid >= 0 and st == 0
                for name in ("info", "pass_len", "pass_dist", "data"):
                    assert np.array_equal(getattr(got, name), getattr(want[which[rid]], name)), name
                eng.release(rid)
            after = eng.stats()
            wide = after["batch_frames"] - before["batch_frames"] > 2 * (after["batches"] - before["batches"])
            if wide:
                break
        assert wide
    finally:
        AT.set_tuning(1, None)
        eng.close()
        dev.close()


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,fk,planar", [(1998, 1080, 0, False), (3996, 2160, 1, True), (2001, 1077, 0, False)])
def test_tile_shapes_give_the_same_coefficients(W, H, fk, planar):
    """Every front-end tile shape (64 x 64, 128 x 64, 64 x 128 at level 1 and at the later
    levels) gives the same X'Y'Z' codes, wavelet planes, quantised words and Tier-1 frame."""
    prof = 1 if fk else 0
    dev = P.Plugin().device(0)
    lay = P.LayoutHolder(W, H, fk)
    if planar:
        fmt, col = P.planar_format(W, H, bits=10, sx=1, sy=0), P.color("pq", "bt2020")
        frame = synth.yuv422p10(W, H, seed=91)
    else:
        fmt, col = P.rgb48_format(W, H), P.color_passthrough()
        frame = synth.xyz12_to_rgb48(synth.xyz12_planes(W, H, seed=91))
    try:
        enc = dev.encoder(lay, fmt, col)
        ref, _, rtaps = enc.encode(frame, debug=True)
        for t1, tn in ((1, 0), (2, 0), (0, 1), (0, 2), (1, 2), (2, 1)):
            AT.set_tuning(prof, {"dwtTile1": t1, "dwtTileN": tn})
            got, _, taps = enc.encode(frame, debug=True)
            for k in ("xyz12", "coeffs"):
                assert np.array_equal(taps[k], rtaps[k]), f"tiles {t1}/{tn}: {k} differ"
            assert np.array_equal(taps["wavelet"].view(np.uint32), rtaps["wavelet"].view(np.uint32)), \
                f"tiles {t1}/{tn}: wavelet planes differ"
            assert np.array_equal(got.info, ref.info) and np.array_equal(got.data, ref.data)
            assert np.array_equal(got.pass_len, ref.pass_len) and np.array_equal(got.pass_dist, ref.pass_dist)
        enc.close()
    finally:
        AT.set_tuning(prof, None)
        dev.close()
