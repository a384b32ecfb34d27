"""The decoder's kernels against the C oracle, at sizes where tiles, stripes and code-blocks are
cut: the picture from the dequantised planes (inverse wavelet, inverse ICT, 12 bits). Bit-identical:
the oracle takes the same float operations in the same order."""
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
