"""The decoder's kernels against the C oracle, at sizes where tiles, stripes and code-blocks are
cut: the dequantised planes from the codewords, sound, cut short and damaged, and the picture
from the planes (inverse wavelet, inverse ICT, 12 bits). Bit-identical: the oracle takes the same
float operations in the same order."""
import numpy as np
import pytest

from libgail_b200 import codestream as CS
from libgail_b200 import plugin as P
from libgail_b200 import synth
from oracle.oracle import Oracle


@pytest.fixture(scope="module")
def dev():
    d = P.Plugin().device(0)
    yield d
    d.close()


def _codestream(dev, w, h, fourk, mbps):
    lay = P.LayoutHolder(w, h, fourk)
    enc = dev.encoder(lay, P.rgb48_format(w, h), P.color_passthrough())
    t1, _, _ = enc.encode(synth.xyz12_to_rgb48(synth.xyz12_planes(w, h, seed=w + h)))
    enc.close()
    return CS.rate_and_build(lay, t1, max_mbps=mbps, comp_mbps=mbps)[0]


def _picture(planes, levels, reduce, high):
    o = Oracle()
    w, h = planes.shape[2], planes.shape[1]
    y = [o.idwt(p, levels, reduce) for p in planes]
    for _ in range(reduce):
        w, h = (w + 1) // 2, (h + 1) // 2
    y0, y1, y2 = (np.ascontiguousarray(p[:h, :w], np.float32) for p in y)
    f = np.float32
    v = np.stack([y0 + f(1.402) * y2, y0 + f(-0.34413) * y1 + f(-0.71414) * y2, y0 + f(1.772) * y1], axis=-1)
    return (np.clip(np.floor(v + f(2048.5)), 0, 4095).astype(np.uint16) << (4 if high else 0)).astype(np.uint16)


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,fourk,reduce,high", [(64, 64, 0, 0, False), (65, 130, 0, 0, True), (131, 67, 1, 0, False),
                                                   (333, 200, 1, 1, False), (1030, 70, 0, 2, False),
                                                   (67, 515, 0, 4, False), (641, 129, 0, 5, True)])
def test_picture_matches_oracle(dev, w, h, fourk, reduce, high):
    cs = _codestream(dev, w, h, fourk, 20.0)
    lay, blocks = CS.parse(cs)
    dec = dev.decoder(lay, reduce=reduce, high_bits=high)
    pic, _, wl = dec.decode(cs, blocks.view(P.CBLK_CODE_DTYPE), frame_layout=lay, wavelet=True)
    dec.close()
    assert np.array_equal(pic, _picture(wl.reshape(3, h, w), 6 if fourk else 5, reduce, high))


def _planes(lay, blocks, data):
    o = Oracle()
    out = np.zeros((3, lay.height, lay.width), np.float32)
    for b in lay.bands:
        half = np.float32(0.5) * np.float32(b.delta)
        for k in range(b.ncbx * b.ncby):
            c = blocks[b.cblkBase + k]
            x, y = 32 * (k % b.ncbx), 32 * (k // b.ncbx)
            w, h = min(32, b.w - x), min(32, b.h - y)
            off, n = int(c["offset"]), int(c["len"])
            if not c["passes"] or not 1 <= c["nbps"] <= 30 or off + n > len(data):
                continue
            words = o.t1_decode(data[off:off + n], w, h, b.orient, int(c["nbps"]), int(c["passes"])).reshape(32, 32)[:h, :w]
            mag = (words & 0x7FFFFFFF).astype(np.float32) * half
            out[b.comp, b.py0 + y:b.py0 + y + h, b.px0 + x:b.px0 + x + w] = np.where(words >> 31, -mag, mag)
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,fourk", [(64, 64, 0), (65, 130, 0), (131, 67, 1), (333, 200, 1)])
@pytest.mark.parametrize("how", ["sound", "cut", "junk", "ff", "wild", "long"])
def test_planes_match_oracle(dev, w, h, fourk, how):
    cs = _codestream(dev, w, h, fourk, 20.0)
    lay, b = CS.parse(cs)
    b = b.view(P.CBLK_CODE_DTYPE).copy()
    rng = np.random.default_rng(w + h)
    data = np.frombuffer(cs, np.uint8).copy()
    if how == "cut":
        b["passes"] = b["passes"] * rng.random(len(b))
    elif how == "junk":
        data = rng.integers(0, 256, len(data), dtype=np.uint8)
    elif how in ("ff", "long"):  # markers, and bytes after 0xFF that carry
        at = np.flatnonzero(rng.random(len(data) - 1) < 0.03)
        data[at] = 0xFF
        data[at + 1] = rng.integers(0x78, 0x98, len(at))
    elif how == "wild":
        b["nbps"], b["passes"] = rng.integers(0, 34, len(b)), rng.integers(0, 100, len(b))
        b["len"], b["offset"] = rng.integers(0, 60, len(b)), rng.integers(0, len(data) + 20, len(b))
    if how == "long":  # codewords longer than the kernel's copy of them
        b["len"] = np.minimum(5000, len(data) - b["offset"].astype(np.int64))
        b["nbps"], b["passes"] = np.where(b["passes"], 22, b["nbps"]), np.where(b["passes"], 64, 0)
    dec = dev.decoder(lay)
    _, _, wl = dec.decode(data.tobytes(), b, frame_layout=lay, wavelet=True)
    dec.close()
    want = _planes(lay, b, data.tobytes())
    assert np.array_equal(wl.reshape(3, h, w).view(np.uint32) & 0x7FFFFFFF, want.view(np.uint32) & 0x7FFFFFFF)
    assert np.array_equal(wl.reshape(3, h, w), want)


@pytest.mark.gpu
def test_insignificant_samples_are_zero_whatever_the_step(dev):
    w, h = 130, 65
    cs = _codestream(dev, w, h, 0, 20.0)
    lay, b = CS.parse(cs)
    b = b.view(P.CBLK_CODE_DTYPE).copy()
    sound = _planes(lay, b, cs)
    for band in lay.bands:
        band.delta = float("inf")
    dec = dev.decoder(lay)
    _, _, wl = dec.decode(cs, b, frame_layout=lay, wavelet=True)
    dec.close()
    zero = sound == 0
    assert 0.01 < zero.mean() < 0.99
    assert not wl.reshape(3, h, w)[zero].any()  # NaN counts as any
    assert not np.isfinite(wl.reshape(3, h, w)[~zero]).any()
