"""A device codestream that turns out to be damaged (its slices are not where
they should be, and following the precinct lengths does not lead to its end
either) is refused after one decode and one look for its precincts, not after
two decodes."""
import ctypes
import time

import numpy as np
import pytest

import jxs_synth as S

pytestmark = pytest.mark.gpu

W, H, D, BPP = 7680, 4320, 12, 2


def test_one_decode(gpu):
    torch = pytest.importorskip("torch")
    planes = S.frame(W, H, D, S.FMT_YUV444, seed=1)
    enc = gpu.Encoder(W, H, D, S.FMT_YUV444, BPP)
    bs = enc.encode(planes)
    enc.close()
    dec = gpu.Decoder(bs)
    outs = [torch.zeros((H, W), dtype=torch.int16, device="cuda") for _ in range(3)]
    ptrs = [(t.data_ptr(), t.shape[1]) for t in outs]
    damaged = bs.copy()
    damaged[-1] ^= 0xff  # no end marker
    dev = [torch.from_numpy(b).cuda() for b in (bs, damaged)]
    frames = [dec.make_frame(b.data_ptr(), ptrs, bs_size=len(bs)) for b in dev]
    torch.cuda.synchronize()
    times = [[], [], []]
    size = ctypes.c_uint32()

    def look():
        return gpu.lib().svt_jpeg_xs_gpu_decoder_locate_frame(ctypes.byref(dec.api), dev[1].data_ptr(), len(bs), ctypes.byref(size),
                                                              None, 0, None)

    for i in range(44):
        for k, f in enumerate(frames):
            t = time.perf_counter()
            assert dec.send_frame(f) == 0
            r, _ = dec.get()
            times[k].append(time.perf_counter() - t)
            assert r == (gpu.E_DEC_INVALID_BITSTREAM if k else 0)
        t = time.perf_counter()
        assert look() == gpu.E_DEC_INVALID_BITSTREAM
        times[2].append(time.perf_counter() - t)
    dec.close()
    good, bad, locate = (float(np.median(t[4:])) for t in times)
    print("good %.1f us, damaged %.1f us, a look for the precincts %.1f us" % (good * 1e6, bad * 1e6, locate * 1e6))
    assert bad < good + locate + good / 4
