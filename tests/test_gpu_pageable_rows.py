"""Decoding one frame at a time to pageable memory: rows on aligned addresses
take no longer than packed ones of the same frame, which start anywhere (the
same bytes cross the link)."""
import time

import numpy as np
import pytest

import jxs_synth as S

pytestmark = pytest.mark.gpu


def rows(shape, dtype, stride):
    raw = np.ones(shape[0] * stride * np.dtype(dtype).itemsize + 64, np.uint8)
    at = -raw.ctypes.data % 64
    return raw[at:at + shape[0] * stride * np.dtype(dtype).itemsize].view(dtype).reshape(shape[0], stride)


def test_aligned_rows_of_16_bit_samples(gpu):
    w, h, d, bpp = 3838, 2160, 10, 3
    enc = gpu.Encoder(w, h, d, S.FMT_YUV422, bpp)
    bs = enc.encode(S.frame(w, h, d, S.FMT_YUV422, seed=1))
    enc.close()
    dec = gpu.Decoder(bs)
    want = dec.decode(bs)
    padded = [rows(x.shape, x.dtype, (x.shape[1] + 31) // 32 * 32) for x in want]
    packed = [rows(x.shape, x.dtype, x.shape[1]) for x in want]
    times = []
    for planes in (packed, padded):
        f = dec.make_frame(bs, [(p.ctypes.data, p.shape[1]) for p in planes])
        for c, p in enumerate(planes):
            f.image.alloc_size[c] = p.nbytes
        t = []
        for _ in range(50):
            a = time.perf_counter()
            assert dec.send_frame(f) == 0
            r, _ = dec.get()
            t.append(time.perf_counter() - a)
            assert r == 0
        times.append(float(np.median(t[10:])))
        assert all(np.array_equal(p[:, :x.shape[1]], x) for p, x in zip(planes, want))
    dec.close()
    print("packed rows %.1f us, aligned rows %.1f us" % (times[0] * 1e6, times[1] * 1e6))
    assert times[1] < 1.1 * times[0]
