"""Performance cases: what users of the codec have it do.

A case is one call, or one encode and decode, of the library on frames of one
shape (or a batch of frames of several), through the entry points a program
calls: send_picture / get_packet, send_frame / get_frame, and the batch form
svt_jpeg_xs_gpu_batch_encode / _decode.  Sizes, formats, bit rates and the
content model are those of the benchmark and the tests.
"""
import ctypes
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "svt-jpeg-xs_gb300"))

import jxs  # noqa: E402

FORMATS = {"420": jxs.FMT_YUV420, "422": jxs.FMT_YUV422, "444": jxs.FMT_YUV444, "rgb": jxs.FMT_PACKED_RGB}

# options of a case that are the encoder's defaults
DEFAULTS = {"v": 2, "h": 5, "quant": 0, "slice": 16, "sig": 1, "rc": 1, "signs": 0, "vpred": 0, "noise": False}


def _case(what, shapes, where="device", **options):
    """what: encode, decode or roundtrip, one frame at a time, or
    batch_encode, batch_decode: all frames in one batch.  shapes: text of
    space-separated frames, each [count*]WIDTHxHEIGHT/format/depth/bpp, the
    bit rate as a fraction NUM:DEN.  where: planes and codestreams in device
    memory or in ordinary (pageable) host memory."""
    c = dict(what=what, shapes=shapes, where=where)
    c.update(DEFAULTS)
    c.update(options)
    return c


MIXED = "16*1280x720/420/8/1:1 16*1920x1080/444/12/4:1 16*3840x2160/rgb/8/2:1"


def listed():
    cases = {
        # the smallest call: a thumbnail-sized frame there and back, all launches and latency
        "small_roundtrip": _case("roundtrip", "256x64/422/8/5:1"),
        # a plugin's call: one HD frame from and to the host memory of a caller that knows nothing of the GPU
        "hd_host_encode": _case("encode", "1920x1080/422/8/5:1", "host"),
        "hd_host_decode": _case("decode", "1920x1080/422/8/5:1", "host"),
        # live contribution: one 4K frame at a time, its latency, in device memory
        "uhd_encode": _case("encode", "3840x2160/422/10/3:1"),
        "uhd_decode": _case("decode", "3840x2160/422/10/3:1"),
        # throughput: 4K frames in batches (the benchmark's stream)
        "uhd_batch_encode": _case("batch_encode", "8*3840x2160/422/10/3:1"),
        "uhd_batch_decode": _case("batch_decode", "8*3840x2160/422/10/3:1"),
        # a server's batch: frames of many streams, three formats and depths, low to middling rates
        "mixed_batch_encode": _case("batch_encode", MIXED),
        "mixed_batch_decode": _case("batch_decode", MIXED),
        # mastering: large 14-bit frames with a quarter of noise, one vertical level
        "8k_batch_encode": _case("batch_encode", "8*7680x4320/444/14/3:2", v=1, noise=True),
        "8k_batch_decode": _case("batch_decode", "8*7680x4320/444/14/3:2", v=1, noise=True),
        # archive settings on an odd size: every coding option on, there and back
        "odd_options_roundtrip": _case("roundtrip", "1279x717/444/12/4:1", quant=1, rc=3, signs=2, vpred=2),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def _log_size(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _draw_shape(rng, most, v, slice_height):
    """One frame's shape of at most `most` luma pixels."""
    fmt = rng.choice(["420", "422", "422", "444", "rgb"])
    w = _log_size(rng, 256, 7680)
    h = max(16, min(4320, most // w, int(w * rng.uniform(0.2, 0.8))))
    if fmt in ("420", "422"):
        w += w % 2
    if fmt == "420":
        h -= h % 2
    depth = rng.choice([8, 8, 10, 10, 12, 14])
    # narrow precincts need the bits for their headers
    least = 2 + 6400 // (w << v)
    num = max(least, rng.choice([1, 2, 3, 4, 5, 6, 8]))
    num = min(num, 1400000 // (w * slice_height))  # a slice of at most 175 kB
    den = 2 if num >= 2 * least and rng.random() < 0.25 else 1
    return "%dx%d/%s/%d/%d:%d" % (w, h, fmt, depth, num, den)


def draw(rng):
    what = rng.choice(["encode", "decode", "encode", "decode", "roundtrip", "batch_encode", "batch_decode"])
    batch = what.startswith("batch")
    options = {"v": rng.choice([1, 2, 2])}
    if rng.random() < 0.3:
        options["quant"] = 1
    if rng.random() < 0.2:
        options["sig"] = 0
    if rng.random() < 0.3:
        options["rc"] = rng.choice([0, 2, 3])
    if rng.random() < 0.2:
        options["signs"] = rng.choice([1, 2])
    if not batch and rng.random() < 0.1:
        options["vpred"] = rng.choice([1, 2])
    if rng.random() < 0.2:
        options["slice"] = rng.choice([8, 32])
    if not batch:
        where = "host" if what != "roundtrip" and rng.random() < 0.25 else "device"
        return _case(what, _draw_shape(rng, 3840 * 2160, options["v"], options.get("slice", 16)), where, **options)
    shapes = []
    for _ in range(rng.choice([1, 1, 2, 3])):
        n = _log_size(rng, 2, 16)
        shapes.append("%d*%s" % (n, _draw_shape(rng, min(3840 * 2160, 40000000 // n), options["v"], options.get("slice", 16))))
    return _case(what, " ".join(shapes), **options)


def _frames(case):
    """(width, height, format, depth, bpp numerator, denominator) of every
    frame, batches of several shapes in an order of their own"""
    out = []
    for text in case["shapes"].split():
        count, _, one = text.rpartition("*")
        size, fmt, depth, bpp = one.split("/")
        w, h = size.split("x")
        num, den = bpp.split(":")
        out += [(int(w), int(h), fmt, int(depth), int(num), int(den))] * int(count or 1)
    random.Random(3).shuffle(out)
    return out


def _component_sizes(w, h, fmt):
    cw, ch = (w // 2 if fmt in ("420", "422") else w), (h // 2 if fmt == "420" else h)
    return [(w, h), (cw, ch), (cw, ch)]


def work(case):
    total = 0
    passes = 2 if case["what"] == "roundtrip" else 1
    for w, h, fmt, depth, num, den in _frames(case):
        samples = sum(a * b for a, b in _component_sizes(w, h, fmt))
        total += samples * (1 if depth <= 8 else 2) + (w * h * num // den + 7) // 8
    return {"bytes": passes * total, "flops": 0}


def _plane(gen, rng, w, h, depth, noise):
    """A gradient over the video range, about Gaussian noise and 20
    rectangles; with `noise` a quarter of uniform noise."""
    dev = "cuda"
    maxv = (1 << depth) - 1
    lo, hi = 16 * maxv // 255, 235 * maxv // 255
    x = torch.arange(w, device=dev, dtype=torch.float32)[None, :] / (2 * max(w - 1, 1))
    y = torch.arange(h, device=dev, dtype=torch.float32)[:, None] / (2 * max(h - 1, 1))
    img = (lo + (hi - lo) * (x + y)).to(torch.int16)
    r = max(1, int(4.0 * maxv / 255.0 * 0.8660254 - 0.5))
    for _ in range(4):
        img += torch.randint(-r, r + 1, (h, w), generator=gen, device=dev, dtype=torch.int16)
    for _ in range(20):
        x0, x1 = sorted(rng.randrange(w) for _ in range(2))
        y0, y1 = sorted(rng.randrange(h) for _ in range(2))
        img[y0:y1 + 1, x0:x1 + 1] = rng.randrange(maxv + 1)
    if noise:
        img[:h // 2, :w // 2] = torch.randint(0, maxv + 1, (h // 2, w // 2), generator=gen, device=dev, dtype=torch.int16)
    img.clamp_(0, maxv)
    return img.to(torch.uint8) if depth <= 8 else img


def _planes(gen, rng, w, h, fmt, depth, noise):
    planes = [_plane(gen, rng, a, b, depth, noise) for a, b in _component_sizes(w, h, fmt)]
    return [torch.stack(planes, dim=-1).reshape(h, 3 * w).contiguous()] if fmt == "rgb" else planes


def _encoder(case, f):
    w, h, fmt, depth, num, den = f
    return jxs.Encoder(w, h, depth, FORMATS[fmt], num, den, case["v"], case["h"], quantization=case["quant"],
                       slice_height=case["slice"], rate_control_mode=case["rc"], coding_significance=case["sig"],
                       coding_signs_handling=case["signs"], coding_vertical_prediction_mode=case["vpred"])


def _pointers(tensors):
    return [(t.data_ptr(), t.shape[1]) for t in tensors]


def _device_frame(codec, planes, codestream):
    if isinstance(codec, jxs.Encoder):
        return codec.make_frame(_pointers(planes), codestream.data_ptr(), codestream.numel())
    return codec.make_frame(codestream.data_ptr(), _pointers(planes), codestream.numel())


def _picture(f, dtype):
    """One buffer for the planes of a decoded frame, and its planes, each on
    a boundary of 256 samples."""
    sizes = _component_sizes(*f[:3])
    starts = [0]
    for a, b in sizes:
        starts.append((starts[-1] + a * b + 255) & ~255)
    buffer = torch.zeros(starts[-1], dtype=dtype, device="cuda")
    return buffer, [buffer[s:s + a * b].view(b, a) for s, (a, b) in zip(starts, sizes)]


def _check(r):
    if r != jxs.E_NONE:
        raise jxs.JxsError("codec", r)


def _one(codec, frame):
    _check(codec.send_frame(frame))
    _check(codec.get()[0])


class State:
    """Handles, buffers and frame structures of one case."""

    def __init__(self, case, seed):
        self.what, self.host = case["what"], case["where"] == "host"
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        rng = random.Random(seed)
        frames = _frames(case)
        # one handle per shape, as a server keeps one per stream
        encoders = {f: _encoder(case, f) for f in frames}
        planes = [_planes(gen, rng, *f[:4], case["noise"]) for f in frames]
        streams = [torch.zeros(encoders[f].frame_bytes, dtype=torch.uint8, device="cuda") for f in frames]
        torch.cuda.synchronize()  # the library works on streams of its own
        self.keep = [encoders, planes, streams]
        self.codecs, self.frames, self.outputs = [], [], []
        encode, decode = self.what.endswith("encode"), self.what.endswith("decode")
        if decode:
            for f, p, s in zip(frames, planes, streams):
                _one(encoders[f], _device_frame(encoders[f], p, s))
        if not encode:
            decoders = {}
            for f, p, s in zip(frames, planes, streams):
                if f not in decoders:
                    if not decode:
                        _one(encoders[f], _device_frame(encoders[f], p, s))
                    decoders[f] = jxs.Decoder(s.cpu().numpy())
            buffers = [_picture(f, p[0].dtype) for f, p in zip(frames, planes)]
            outs = [views for _, views in buffers]
            self.keep += [decoders, outs]
        if self.host:
            (f,), planes, streams = frames, [t.cpu().numpy() for t in planes[0]], streams[0].cpu().numpy()
            if encode:
                self.codecs, self.outputs = [encoders[f]], streams
                self.frames = [encoders[f].make_frame(planes, streams)]
            else:
                self.outputs = [t.cpu().numpy() for t in outs[0]]
                self.codecs, self.frames = [decoders[f]], [decoders[f].make_frame(streams, self.outputs)]
            self.keep += [planes, streams]
            return
        if not decode:
            self.codecs += [encoders[f] for f in frames]
            self.frames += [_device_frame(encoders[f], p, s) for f, p, s in zip(frames, planes, streams)]
            self.outputs += streams
        if not encode:
            self.codecs += [decoders[f] for f in frames]
            self.frames += [_device_frame(decoders[f], o, s) for f, o, s in zip(frames, outs, streams)]
            self.outputs += [buffer for buffer, _ in buffers]
        if self.what.startswith("batch"):
            samples = sum(sum(a * b for a, b in _component_sizes(*f[:3])) for f in frames)
            self.batch = jxs.Batch(20 * samples + (len(frames) << 22))
            n = len(frames)
            self.handles = (ctypes.c_void_p * n)(*[ctypes.addressof(c.api) for c in self.codecs])
            self.pointers = (ctypes.c_void_p * n)(*[ctypes.addressof(f) for f in self.frames])
        torch.cuda.synchronize()


def prepare(case, seed):
    return State(case, seed)


def run(state):
    if state.what.startswith("batch"):
        call = jxs.lib().svt_jpeg_xs_gpu_batch_encode if state.what == "batch_encode" else jxs.lib().svt_jpeg_xs_gpu_batch_decode
        _check(call(state.batch.h, state.handles, state.pointers, len(state.frames), None))
        _check(state.batch.wait()[0])
    else:
        for codec, frame in zip(state.codecs, state.frames):
            _one(codec, frame)
    return state.outputs
