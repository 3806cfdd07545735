"""Results for pageable memory: frames one at a time (written in place by the
kernels after a few of them, where the memory allows it) and several in flight,
at any alignment and pitch, in touched and untouched buffers, without a byte
outside the planes or past the codestream."""
import numpy as np
import pytest

import jxs_synth as S

pytestmark = pytest.mark.gpu


def buffer(nbytes, offset, touched):
    raw = np.empty(nbytes + 4096 + offset, np.uint8)
    start = -raw.ctypes.data % 64 + offset
    if touched:
        raw[:] = 0xA5
    return raw, raw[start:start + nbytes]


@pytest.mark.parametrize("w,h,fmt,d,pad,offset", [(640, 64, S.FMT_YUV422, 8, 0, 0), (640, 50, S.FMT_YUV444, 10, 8, 16),
                                                  (321, 33, S.FMT_YUV444, 8, 0, 1), (330, 40, S.FMT_YUV420, 10, 3, 2)])
def test_results_in_pageable_memory(gpu, oracle, w, h, fmt, d, pad, offset):
    planes = S.frame(w, h, d, fmt, seed=5)
    p = oracle.make_params(w, h, d, fmt, 6, 1, 1, 5)
    err, bs = oracle.oracle_encode(p, planes)[:2]
    assert err == 0
    err, want = oracle.oracle_decode(bs)
    assert err == 0
    enc, dec = gpu.Encoder(w, h, d, fmt, 6, 1, 1, 5), gpu.Decoder(bs)
    size = want[0].itemsize
    for flight in (1, 1, 1, 1, 1, 1, 1, 3, 1, 1):
        for touched in (True, False):
            jobs = []
            for _ in range(flight):
                raw, out = buffer(len(bs) + 64, offset, touched)
                outs = [buffer(x.shape[0] * (x.shape[1] + pad) * size, offset, touched) for x in want]
                jobs.append((raw, out, outs))
                assert enc.send(planes, out) == 0
                assert dec.send(bs, [(b.ctypes.data, x.shape[1] + pad) for (_, b), x in zip(outs, want)]) == 0
            for raw, out, outs in jobs:
                r, f = enc.get()
                assert r == 0 and f.bitstream.used_size == len(bs)
                assert np.array_equal(out[:len(bs)], bs)
                assert not touched or (out[len(bs):] == 0xA5).all()
                assert dec.get()[0] == 0
                for (whole, b), x in zip(outs, want):
                    got = b.view(x.dtype).reshape(x.shape[0], x.shape[1] + pad)
                    assert np.array_equal(got[:, :x.shape[1]], x)
                    if touched:
                        got[:, :x.shape[1]] = np.frombuffer(b"\xa5" * size, x.dtype)[0]
                        assert (whole == 0xA5).all()
    enc.close()
    dec.close()


def test_refused_codestreams_between_good_ones(gpu, oracle):
    """A host codestream whose precincts or header are found wrong is refused
    by the host, with its copy to the device already under way."""
    w, h, fmt, d = 640, 64, S.FMT_YUV422, 8
    p = oracle.make_params(w, h, d, fmt, 6, 1, 2, 5)
    err, bs = oracle.oracle_encode(p, S.frame(w, h, d, fmt, seed=5))[:2]
    assert err == 0
    err, want = oracle.oracle_decode(bs)
    assert err == 0
    slice1 = bs.tobytes().index(b"\xff\x20\x00\x04\x00\x01")
    dec = gpu.Decoder(bs)
    for at in (None, None, slice1 + 5, None, slice1 + 6, None, 20, None):
        sent = bs.copy()
        if at is not None:
            sent[at] ^= 0xff
        outs = [np.zeros(x.shape, x.dtype) for x in want]
        r = dec.send(sent, outs)
        r = r or dec.get()[0]
        assert (r != 0) == (at is not None)
        assert r or all(np.array_equal(a, b) for a, b in zip(outs, want))
    dec.close()
