"""Plain decoders beside others and beside encoders, a thread each: every picture is the one its
codestream gives on a GPU of its own, whatever SMs a decode's warps find free."""
import threading

import numpy as np
import pytest

from libgail_b200 import codestream as CS
from libgail_b200 import plugin as P
from libgail_b200 import synth


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,fourk,threads,encoders", [(3996, 2160, 1, 2, 0), (1998, 1080, 0, 4, 0), (1998, 1080, 0, 1, 3)])
def test_decoders_side_by_side(w, h, fourk, threads, encoders):
    dev = P.Plugin().device(0)
    lay = P.LayoutHolder(w, h, fourk)
    enc = dev.encoder(lay, P.rgb48_format(w, h), P.color_passthrough())
    streams = []
    for seed in (1, 2):
        frame = synth.xyz12_to_rgb48(synth.xyz12_planes(w, h, seed=seed))
        cs = CS.rate_and_build(lay, enc.encode(frame)[0], 24.0)[0]
        streams.append((cs, CS.parse(cs)[1].view(P.CBLK_CODE_DTYPE)))
    enc.close()
    encs = [dev.encoder(lay, P.rgb48_format(w, h), P.color_passthrough()) for _ in range(encoders)]
    decoders = [dev.decoder(lay) for _ in range(threads)]
    want = [decoders[0].decode(*s)[0].copy() for s in streams]
    wrong, failed, done = [], [], threading.Event()

    def work(t):
        pic = np.zeros_like(want[0])
        try:
            for i in range(40):
                k = (i + t) % 2  # never the picture this decoder made before
                decoders[t].decode(*streams[k], out=pic)
                if not np.array_equal(pic, want[k]):
                    wrong.append((t, i, int((pic != want[k]).sum())))
        except Exception as e:  # noqa: BLE001
            failed.append(e)

    def load(e):
        while not done.is_set():
            e.encode(frame)

    loads = [threading.Thread(target=load, args=(e,)) for e in encs]
    ts = [threading.Thread(target=work, args=(t,)) for t in range(threads)]
    for t in loads + ts:
        t.start()
    for t in ts:
        t.join()
    done.set()
    for t in loads:
        t.join()
    for d in decoders + encs:
        d.close()
    dev.close()
    assert not failed, failed
    assert not wrong, wrong[:10]
