"""The transform kernels at the edges of their strips and chunks: widths and
heights around the boundaries of the work split, every level count, sample
size and layout, against the oracle byte for byte."""
import numpy as np
import pytest

import jxs_synth as S

pytestmark = pytest.mark.gpu


def check(gpu, oracle, w, h, d, fmt, v, hh, bpp):
    planes = S.frame(w, h, d, fmt, seed=w * 7 + h)
    p = oracle.make_params(w, h, d, fmt, bpp, 1, v, hh)
    err, ref_bs = oracle.oracle_encode(p, planes)[:2]
    assert err == 0
    enc = gpu.Encoder(w, h, d, fmt, bpp, 1, v, hh)
    bs = enc.encode(planes)
    enc.close()
    assert np.array_equal(bs, ref_bs)
    dec = gpu.Decoder(ref_bs)
    out = dec.decode(ref_bs)
    dec.close()
    err, want = oracle.oracle_decode(ref_bs)
    assert err == 0 and all(np.array_equal(a, b) for a, b in zip(out, want))


# rows of the horizontal-only levels: 480, 448 or 384 columns per chunk
# forward, 480 or 448 inverse
@pytest.mark.parametrize("w", [383, 384, 385, 447, 448, 449, 479, 480, 481, 511, 512, 513, 897, 961, 1000])
@pytest.mark.parametrize("v,hh", [(0, 5), (0, 4), (0, 3), (0, 1), (1, 5), (1, 3), (1, 2), (1, 1)])
def test_horizontal_only_chunks(gpu, oracle, w, v, hh):
    check(gpu, oracle, w << v, 4 << v, 10 if w & 1 else 8, S.FMT_YUV444, v, hh, 8)


@pytest.mark.parametrize("w", [4 * 480 - 4, 4 * 480, 4 * 480 + 4, 4 * 480 + 6])
def test_horizontal_only_chunks_two_vertical_levels(gpu, oracle, w):
    check(gpu, oracle, w, 10, 12, S.FMT_YUV420, 2, 5, 6)
