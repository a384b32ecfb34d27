"""The work a user of this codec has it do, as cases to time and compare.

Every case goes through a public entry point of the package, from what a program holds before
the call (a frame in the encoder's input buffer or on the GPU, a codestream in memory, a batch of
code-blocks) to what it gets back (the packed Tier-1 frame, a codestream, a picture). Five kinds:

  encode        one frame through the plugin's encoder_encode (plugin.Encoder), as libgail drives
                it: the frame already in the encoder's pinned input buffer, the Tier-1 frame
                taken out of the encoder's output buffers
  decode        one codestream, parsed and decoded (codestream.parse, plugin.Decoder)
  serve_encode  several frames through the served engine to their DCI codestreams
  serve_decode  several codestreams through the served engine to their pictures
  blocks        a batch of code-blocks through t1_encode_blocks

Outputs are bytes and whole numbers, and the library's contract is that they are the same
whatever the launch shapes, so every case is compared exactly and none has a 64-bit counterpart.
"""
from __future__ import annotations

import ctypes as C
import math
import os

import numpy as np
import torch

import libgail_b200 as gb
from libgail_b200 import autotune
from libgail_b200 import codestream as cs
from libgail_b200 import plugin as P
from libgail_b200.engine import Engine

TUNING = os.path.join(os.path.dirname(os.path.abspath(gb.__file__)), "tuning_b200.json")
FPS = 24.0

# Colour settings by name: X'Y'Z' input as it is, SDR BT.709, PQ BT.2020, HLG BT.2020 through the
# shoulder tone map and the P3-D65 gamut compression.
COLORS = ("xyz", "bt709", "pq", "hlg_managed")
# Frame formats by name: (planar, bits, chroma shift x, chroma shift y).
FORMATS = {"rgb48": (False, 16, 0, 0), "422p10": (True, 10, 1, 0), "420p8": (True, 8, 1, 1),
           "420p10": (True, 10, 1, 1), "444p12": (True, 12, 0, 0)}


def listed():
    return [
        # the headline workload's frame, one at a time: 4K HDR broadcast or mezzanine material
        {"name": "encode_4k_pq", "kind": "encode", "w": 3996, "h": 2160, "fmt": "422p10", "color": "pq", "early": False},
        # a 2K flat digital cinema master, X'Y'Z' already
        {"name": "encode_2k_xyz", "kind": "encode", "w": 1998, "h": 1080, "fmt": "rgb48", "color": "xyz", "early": False},
        # gail.h's default encode: Tier-1 stops early at 0.25 of the last frame's threshold
        {"name": "encode_2k_early", "kind": "encode", "w": 2048, "h": 858, "fmt": "420p8", "color": "bt709", "early": True},
        # an odd size, full chroma, through the tone map and the gamut compression
        {"name": "encode_ragged_hlg", "kind": "encode", "w": 1283, "h": 717, "fmt": "444p12", "color": "hlg_managed", "early": False},
        # the smallest frame the codec takes: launches and latency
        {"name": "encode_min", "kind": "encode", "w": 64, "h": 64, "fmt": "rgb48", "color": "xyz", "early": False},
        # playback of a 4K package at the DCI peak rate, and of a 2K one at half size (a preview)
        {"name": "decode_4k", "kind": "decode", "w": 3996, "h": 2160, "reduce": 0, "bpp": 1.207, "high": False},
        {"name": "decode_2k_half", "kind": "decode", "w": 1998, "h": 1080, "reduce": 1, "bpp": 4.827, "high": False},
        # a small odd picture with the codes in the high bits
        {"name": "decode_small", "kind": "decode", "w": 333, "h": 241, "reduce": 0, "bpp": 3.0, "high": True},
        # the served engine: 4K frames resident on the GPU, 2K frames from pinned host memory
        {"name": "serve_encode_4k", "kind": "serve_encode", "w": 3996, "h": 2160, "fmt": "422p10", "color": "pq", "frames": 24, "device": True},
        {"name": "serve_encode_2k", "kind": "serve_encode", "w": 1998, "h": 1080, "fmt": "rgb48", "color": "xyz", "frames": 32, "device": False},
        # several codestreams at once (a review server)
        {"name": "serve_decode_4k", "kind": "serve_decode", "w": 3996, "h": 2160, "reduce": 0, "bpp": 1.207, "frames": 8},
        # a caller with its own wavelet: a few code-blocks at a time
        {"name": "blocks_64", "kind": "blocks", "n": 64, "planes": 10},
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["encode"] * 4 + ["decode"] * 3 + ["serve_encode", "serve_decode", "blocks"])
    if kind == "blocks":
        return {"kind": kind, "n": _log_size(rng, 1, 2048), "planes": rng.randint(2, 14)}
    w, h = _log_size(rng, 64, 4096), _log_size(rng, 64, 2160)
    if kind == "encode":
        return {"kind": kind, "w": w, "h": h, "fmt": rng.choice(sorted(FORMATS)), "color": rng.choice(COLORS),
                "early": rng.random() < 0.25}
    if kind == "decode":
        return {"kind": kind, "w": w, "h": h, "reduce": rng.choice([0, 0, 0, 1, 2]), "bpp": round(rng.uniform(0.4, 5.0), 3),
                "high": rng.random() < 0.3}
    n = rng.randint(2, 12)
    if kind == "serve_encode":
        return {"kind": kind, "w": w, "h": h, "fmt": rng.choice(sorted(FORMATS)), "color": rng.choice(COLORS), "frames": n,
                "device": rng.random() < 0.5}
    return {"kind": kind, "w": w, "h": h, "reduce": rng.choice([0, 0, 1]), "bpp": round(rng.uniform(0.4, 5.0), 3),
            "frames": min(n, 8)}


# ------------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _plane(w, h, g):
    """One plane of 12-bit picture content on the GPU, with the statistics of synth.plane: a smooth
    pattern, 25 rectangles with hard edges, and grain."""
    u = torch.rand(3 + 5 * 25, generator=g, device="cuda").cpu().tolist()
    x = torch.arange(w, device="cuda", dtype=torch.float32)
    y = torch.arange(h, device="cuda", dtype=torch.float32)
    sx = 900.0 * torch.sin(2 * math.pi * (1 + 5 * u[0]) * x / w + 2 * math.pi * u[2])
    cy = torch.cos(2 * math.pi * (1 + 5 * u[1]) * y / h)
    v = torch.randn((h, w), generator=g, device="cuda") * 30.0 + 2048.0 + cy[:, None] * sx[None, :]
    for k in range(25):
        a = u[3 + 5 * k: 8 + 5 * k]
        rw, rh = int(w / 40 + a[0] * (w / 4 - w / 40)), int(h / 40 + a[1] * (h / 4 - h / 40))
        x0, y0 = int(a[2] * (w - rw)), int(a[3] * (h - rh))
        v[y0:y0 + rh, x0:x0 + rw] += -600 + 1200 * a[4]
    return v.round_().clamp_(0, 4095)


def _frame(case, g):
    """The frame's bytes as the encoder takes them: a flat uint8 tensor on the GPU."""
    w, h = case["w"], case["h"]
    planar, bits, sx, sy = FORMATS[case["fmt"]]
    if not planar:
        v = torch.stack([_plane(w, h, g) for _ in range(3)], dim=-1).to(torch.int32)
        return ((v * 65535 + 2047) // 4095).to(torch.uint16).view(torch.uint8).reshape(-1)
    cw, ch = (w + sx) >> sx, (h + sy) >> sy
    scale = float(1 << (bits - 8))
    parts = []
    for k, (pw, ph) in enumerate(((w, h), (cw, ch), (cw, ch))):
        v = (_plane(pw, ph, g) * ((219 if k == 0 else 224) * scale / 4095.0) + 16 * scale).round_()
        parts.append((v.to(torch.uint8) if bits == 8 else v.to(torch.int32).to(torch.uint16)).reshape(-1).view(torch.uint8))
    return torch.cat(parts)


def _format(case):
    planar, bits, sx, sy = FORMATS[case["fmt"]]
    if not planar:
        return P.rgb48_format(case["w"], case["h"])
    return P.planar_format(case["w"], case["h"], bits=bits, sx=sx, sy=sy)


def _color(name):
    if name == "xyz":
        return P.color_passthrough()
    if name == "bt709":
        return P.color("bt1886", "bt709")
    if name == "pq":
        return P.color("pq", "bt2020")
    return P.color_managed("hlg", "bt2020", tone_map="shoulder", tone_norm="maxrgb", gamut="p3d65")


def _layout(case):
    return P.LayoutHolder(case["w"], case["h"], int(case["w"] > 2048 or case["h"] > 1080))


def _mbps(case):
    """The rate cap that leaves `bpp` codestream bits per pixel (and room for the headers of the
    smallest pictures)."""
    return max(case["bpp"] * case["w"] * case["h"], 80000.0) * FPS / 1e6


# ------------------------------------------------------------------------ handles
class Handle:
    """Something with a close(), closed when its last user is gone."""

    def __init__(self, obj, *more):
        self.obj, self.more = obj, more

    def __del__(self):
        for o in (self.obj, *self.more):
            o.close()


_program = {}  # what a program makes once: the device, the tuning, the handle used last


def _device():
    if "dev" not in _program:
        # the tuning file, applied when the program starts, as bench.py and serve_mix do
        _program["policy"] = autotune.apply(TUNING, device_name=torch.cuda.get_device_name(0))
        _program["dev"] = P.Plugin().device(0)
    return _program["dev"]


def _kept(key, make):
    """The program's handle for `key`; one is kept, so that new inputs of the same sort find it."""
    if _program.get("key") != key:
        _program["handle"] = None
        _program["handle"] = Handle(*make())
        _program["key"] = key
    return _program["handle"]


def _streams(case, g, count):
    """Codestreams of new X'Y'Z' pictures at the case's rate."""
    fcase = dict(case, fmt="rgb48")
    lay = _layout(case)
    h = _kept(("streams", case["w"], case["h"]), lambda: (_device().encoder(lay, _format(fcase), _color("xyz")),))
    out = []
    for _ in range(count):
        f = _frame(fcase, g).cpu().numpy()
        t1, _, _ = h.obj.encode(f)
        out.append(cs.rate_and_build(lay, t1, FPS, _mbps(case), _mbps(case), tag="b200")[0])
    return out


class Taken:
    """A result of varying length, taken out of the library's buffer (which the next call reuses)
    into the program's own, zero past its end."""

    def __init__(self, capacity, dtype):
        self.buf, self.used = torch.zeros(max(1, capacity), dtype=dtype), 0

    def take(self, ptr, count):
        if count > len(self.buf):
            raise RuntimeError(f"{count} values in a buffer of {len(self.buf)}")
        nbytes = count * self.buf.element_size()
        if nbytes >= 4 << 20:  # tens of MB, on several cores
            self.buf[:count].copy_(torch.frombuffer((C.c_uint8 * nbytes).from_address(ptr), dtype=self.buf.dtype))
        elif nbytes:
            C.memmove(self.buf.data_ptr(), ptr, nbytes)
        if self.used > count:
            self.buf[count:self.used].zero_()
        self.used = count
        return self.buf


def _view(ptr, nbytes, dtype, owner):
    """The library's buffer as an array that keeps `owner` (whose buffer it is) alive."""
    buf = (C.c_uint8 * nbytes).from_address(ptr)
    buf.owner = owner
    return np.frombuffer(buf, dtype)


def _address(p):
    return C.cast(p, C.c_void_p).value


# ------------------------------------------------------------------------ the cases
class Encode:
    def __init__(self, case, seed):
        lay = _layout(case)
        self.handle = Handle(_device().encoder(lay, _format(case), _color(case["color"])))
        enc = self.enc = self.handle.obj
        f = _frame(case, _gen(seed)).cpu().numpy()
        self.buf = enc.input_buffer()
        C.memmove(self.buf, f.ctypes.data, f.nbytes)
        if case["early"]:  # the threshold libgail's pipeline takes from the frame before
            t1, _ = enc.encode_view(self.buf)
            bpp = 2.3e8 / FPS / (3996 * 2160) if lay.fourk else 2.3e8 / FPS / (1998 * 1080)
            rate = _mbps(dict(case, bpp=bpp))
            enc.set_slope(0.25 * cs.rate_and_build(lay, t1, FPS, rate, rate)[2])
        n = lay.num_cblks
        self.info, self.len, self.dist = Taken(5 * n, torch.int32), Taken(64 * n, torch.int32), Taken(64 * n, torch.int32)
        self.data = Taken(6 * case["w"] * case["h"] + (64 << 10), torch.uint8)

    def run(self):
        t, _ = self.enc.encode_view(self.buf)
        return {"info": self.info.take(_address(t.info), 5 * t.numInfo), "pass_len": self.len.take(_address(t.passLen), t.numPasses),
                "pass_dist": self.dist.take(_address(t.passDist), t.numPasses), "data": self.data.take(_address(t.data), t.numData)}


class Decode:
    def __init__(self, case, seed):
        self.cs, = _streams(case, _gen(seed), 1)
        lay = _layout(case)
        self.handle = Handle(_device().decoder(lay, reduce=case["reduce"], high_bits=case["high"]))
        self.dec = self.handle.obj
        self.picture = np.zeros((self.dec.out_h, self.dec.out_w, 3), np.uint16)

    def run(self):
        lay, blocks = cs.parse(self.cs)
        self.dec.decode(self.cs, blocks.view(P.CBLK_CODE_DTYPE), frame_layout=lay, out=self.picture)
        return self.picture


class ServeEncode:
    def __init__(self, case, seed):
        key = tuple(sorted((k, v) for k, v in case.items() if k in ("w", "h", "fmt", "color", "frames")))

        def make():
            _device()
            pol = _program["policy"]
            eng = Engine(0, 0, max_batch=pol["maxBatch"])
            eng.set_policy(pol["maxBatch"], pol["minBatchPct"], pol["maxWaitMs"])
            cls, _ = eng.add_encoder(_layout(case), _format(case), _color(case["color"]))
            eng.reserve(cls, case["frames"])
            eng.set_codestream(fps=FPS, tag="b200", threads=max(2, min(12, (os.cpu_count() or 4) - 2)))
            return (eng,)

        self.handle = _kept(("serve_encode", key), make)
        g = _gen(seed)
        self.frames = [_frame(case, g) for _ in range(case["frames"])]
        if not case["device"]:
            self.frames = [f.cpu().pin_memory() for f in self.frames]
        limit, _ = cs.dci_limits(FPS)
        self.out = [Taken(limit, torch.uint8) for _ in self.frames]

    def run(self):
        eng = self.handle.obj
        at = {eng.submit(0, f): i for i, f in enumerate(self.frames)}
        out = [None] * len(at)
        for _ in range(len(at)):
            rid, _, _, status = eng.wait(60000, copy=False)
            if rid < 0 or status != 0:
                raise RuntimeError(f"request {rid}: status {status}")
            (p, n), _ = eng.codestream(rid, copy=False)
            out[at[rid]] = self.out[at[rid]].take(_address(p), n)
            eng.release(rid)
        return out


class ServeDecode:
    def __init__(self, case, seed):
        self.streams = _streams(case, _gen(seed), case["frames"])
        _device()
        self.handle = Handle(Engine(0, 0))
        self.cls, _ = self.handle.obj.add_decoder(_layout(case), reduce=case["reduce"])
        self.held = []

    def run(self):
        eng = self.handle.obj
        for rid in self.held:  # the pictures of the pass before have been used
            eng.release(rid)
        at = {eng.submit_decode(self.cls, c): i for i, c in enumerate(self.streams)}
        self.held = list(at)
        out = [None] * len(at)
        for _ in range(len(at)):
            rid, _, _, status = eng.wait(60000, copy=False)
            if rid < 0 or status != 0:
                raise RuntimeError(f"request {rid}: status {status}")
            p = eng.picture(rid, copy=False)
            out[at[rid]] = _view(p.ctypes.data, p.nbytes, np.uint16, self.handle).reshape(p.shape)
        return out


class Blocks:
    def __init__(self, case, seed):
        n, planes = case["n"], case["planes"]
        g = _gen(seed)
        # wavelet coefficients: two-sided exponential magnitudes, of `planes` bit-planes at the most
        # (6 fraction bits below them), a third of the blocks clipped at a band's edge
        scale = 2.0 ** (planes + 6) / 12
        m = (-torch.log(torch.rand((n, 1024), generator=g, device="cuda").clamp_min(1e-30)) * scale).clamp_max(2.0 ** (planes + 6) - 1)
        m = m * torch.rand((n, 1), generator=g, device="cuda")
        s = torch.rand((n, 1024), generator=g, device="cuda") < 0.5
        q = m.to(torch.int64)
        q = q + ((s & (q >= 64)).to(torch.int64) << 31)
        self.coeffs = q.cpu().numpy().astype(np.uint32)
        r = torch.rand((n, 4), generator=g, device="cuda").cpu().numpy()
        edge = r[:, 0] < 1 / 3
        self.geom = np.stack([np.where(edge, 1 + (r[:, 1] * 32).astype(np.int32), 32),
                              np.where(edge, 1 + (r[:, 2] * 32).astype(np.int32), 32),
                              (r[:, 3] * 4).astype(np.int32), np.full(n, 64)], axis=1).astype(np.int32)
        self.capacity = n * 160 * (planes + 2)

    def run(self):
        info, plen, pdist, words = gb.t1_encode_blocks(self.coeffs, self.geom)
        data = np.zeros(self.capacity, np.uint8)
        joined = np.frombuffer(b"".join(words), np.uint8)
        data[:len(joined)] = joined
        coded = np.arange(64) < info[:, 1:2]  # the tables are not written past a block's passes
        return {"info": info.view(np.int32), "pass_len": np.where(coded, plen, 0).view(np.int32),
                "pass_dist": np.where(coded, pdist, 0), "data": data}


KINDS = {"encode": Encode, "decode": Decode, "serve_encode": ServeEncode, "serve_decode": ServeDecode, "blocks": Blocks}


def prepare(case, seed):
    return KINDS[case["kind"]](case, seed)


def run(state):
    return state.run()


def work(case):
    """Bytes in and out of one pass: the frame or codestream, and the Tier-1 frame (on this content
    about 2.9 bytes a pixel with every pass), the codestream or the picture."""
    if case["kind"] == "blocks":
        return {"bytes": case["n"] * (4096 + 16 + 16 + 64 * 8 + 70 * case["planes"]), "flops": 0}
    px = case["w"] * case["h"]
    if case["kind"] in ("encode", "serve_encode"):
        planar, bits, sx, sy = FORMATS[case["fmt"]]
        frame = px * 6 if not planar else (px + 2 * ((case["w"] + sx) >> sx) * ((case["h"] + sy) >> sy)) * (1 if bits == 8 else 2)
        if case["kind"] == "encode":
            return {"bytes": frame + 2.9 * px, "flops": 0}
        return {"bytes": case["frames"] * (frame + min(1.2e6, 2.0 * px)), "flops": 0}
    picture = 6 * -(-case["w"] // (1 << case["reduce"])) * -(-case["h"] // (1 << case["reduce"]))
    return {"bytes": case.get("frames", 1) * (picture + case["bpp"] * px / 8), "flops": 0}


def tolerance(case):
    return "exact"
