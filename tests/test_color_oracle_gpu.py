"""The direct colour route's X'Y'Z' codes against the C oracle: every transfer function it has, linear
values far out of range and beyond a float's (where the encoder divides by the reference white's
constant instead of multiplying by its reciprocal), and planar formats of every subsampling, bit
depth and range, whose divisions have reciprocals of their own. Codes are whole numbers, so they
are compared exactly."""
import numpy as np
import pytest

from libgail_b200 import plugin as P
from oracle.oracle import Oracle, Planar

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    d = P.Plugin().device(0)
    yield d
    d.close()


def _codes(dev, w, h, fmt, col, frame):
    enc = dev.encoder(P.LayoutHolder(w, h, 0), fmt, col)
    taps = enc.encode(frame, debug=True)[2]
    enc.close()
    return taps["xyz12"].reshape(h, w, 3)


@pytest.mark.parametrize("transfer,primaries,white", [
    ("bt1886", "bt709", 48.0), ("srgb", "p3d65", 48.0), ("pq", "bt2020", 48.0), ("linear", "dcip3", 52.37),
    ("gamma26", "xyz", 48.0), ("linear", "bt709", 1e-30), ("linear", "bt709", 9e29), ("linear", "bt709", 1e33),
    ("bt1886", "bt709", 1e45), ("linear", "bt709", 1e39)])
def test_values_match_oracle(dev, transfer, primaries, white):
    w, h = 197, 70
    rng = np.random.default_rng(4)
    frame = rng.integers(0, 65536, (h, w, 3)).astype(np.uint16)
    frame[:20] = rng.integers(0, 300, (20, w, 3))
    frame[20:24] = np.arange(4 * w).reshape(4, w, 1) * 83 % 65536  # greys
    got = _codes(dev, w, h, P.rgb48_format(w, h), P.color(transfer, primaries, white), frame)
    want = Oracle().color_frame(frame, P.TRANSFER[transfer], P.PRIMARIES[primaries], white)[1]
    assert np.array_equal(got, want)


@pytest.mark.parametrize("sx,sy", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("bits,full,rgb,chroma", [(8, False, False, 0), (8, True, False, 1), (9, True, False, 2), (10, False, False, 1),
                                                  (12, True, True, 0), (13, True, False, 0), (16, False, False, 2)])
def test_planar_formats_match_oracle(dev, sx, sy, bits, full, rgb, chroma):
    w, h, aw, ah = 131, 96, 125, 81  # a letterbox, odd sizes
    cw, ch = (aw + sx) >> sx, (ah + sy) >> sy
    rng = np.random.default_rng(bits)
    frame = rng.integers(0, 1 << bits, aw * ah + 2 * cw * ch).astype(np.uint8 if bits == 8 else np.uint16)
    fmt = P.planar_format(w, h, bits=bits, sx=sx, sy=sy, chroma=chroma, full_range=full, rgb=rgb, active=(aw, ah))
    got = _codes(dev, w, h, fmt, P.color("bt1886", "bt2020"), frame)
    o = Oracle()
    planar = Planar(width=w, height=h, active_w=aw, active_h=ah, ox=(w - aw) // 2, oy=(h - ah) // 2, sx=sx, sy=sy, rgb=int(rgb),
                    bits=bits, full_range=int(full), chroma=chroma, kr=0.2627, kb=0.0593)
    want = o.color_frame(o.planar_to_rgb48(planar, frame), P.TRANSFER["bt1886"], P.PRIMARIES["bt2020"])[1]
    assert np.array_equal(got, want)
