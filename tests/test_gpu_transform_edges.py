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


# vertical levels: strips of 240 columns and up to 8 row pairs; widths that
# are and are not whole groups of 8 columns, all layouts, both widths of the
# integer lifting (depths up to 12, and 14)
@pytest.mark.parametrize("w,h", [(232, 2), (239, 3), (240, 4), (241, 31), (248, 17), (255, 9), (479, 33), (480, 16), (488, 5), (723, 34)])
@pytest.mark.parametrize("fmt,d", [(S.FMT_YUV444, 8), (S.FMT_YUV444, 12), (S.FMT_YUV444, 14), (S.FMT_PACKED_RGB, 8),
                                   (S.FMT_PACKED_RGB, 12), (S.FMT_PACKED_RGB, 14)])
@pytest.mark.parametrize("v", [1, 2])
def test_vertical_strips(gpu, oracle, w, h, fmt, d, v):
    check(gpu, oracle, w, max(h, 1 << v), d, fmt, v, 5, 14)


@pytest.mark.parametrize("fmt,d", [(S.FMT_YUV422, 8), (S.FMT_YUV422, 10), (S.FMT_PACKED_RGB, 8), (S.FMT_PACKED_RGB, 10)])
@pytest.mark.parametrize("offset,pad", [(0, 1), (1, 0), (3, 5), (0, 16)])
def test_unaligned_device_rows(gpu, oracle, fmt, d, offset, pad):
    """Device planes whose rows start anywhere, samples with bits above the
    depth: read and written sample by sample, nothing outside the rows."""
    torch = pytest.importorskip("torch")
    w, h = 500, 22
    planes = S.frame(w, h, d, fmt, seed=5)
    p = oracle.make_params(w, h, d, fmt, 5, 1, 2, 5)
    err, ref_bs = oracle.oracle_encode(p, planes)[:2]
    assert err == 0

    def padded(a, fill):
        big = np.full(offset + a.shape[0] * (a.shape[1] + pad), fill, a.dtype)
        view = big[offset:].reshape(a.shape[0], a.shape[1] + pad)[:, :a.shape[1]]
        view[:] = a
        return torch.from_numpy(big.view(np.int16) if d > 8 else big).cuda(), big

    size = 1 if d <= 8 else 2
    src = [padded(a | (0x8000 if d > 8 else 0), 0xff)[0] for a in planes]
    enc = gpu.Encoder(w, h, d, fmt, 5, 1, 2, 5)
    out = torch.zeros(enc.frame_bytes, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert enc.send([(t.data_ptr() + offset * size, a.shape[1] + pad) for t, a in zip(src, planes)], out.data_ptr(),
                    out_cap=enc.frame_bytes) == 0
    r, f = enc.get()
    enc.close()
    assert r == 0 and np.array_equal(out.cpu().numpy(), ref_bs)
    err, want = oracle.oracle_decode(ref_bs)
    dec = gpu.Decoder(ref_bs)
    dst = [padded(np.zeros_like(a), 0x5a) for a in want]
    torch.cuda.synchronize()
    assert dec.send(out.data_ptr(), [(t.data_ptr() + offset * size, a.shape[1] + pad) for (t, _), a in zip(dst, want)],
                    bs_size=len(ref_bs)) == 0
    r, _ = dec.get()
    dec.close()
    assert err == 0 and r == 0
    for (t, big), a in zip(dst, want):
        expect = big.copy()
        expect[offset:].reshape(a.shape[0], a.shape[1] + pad)[:, :a.shape[1]] = a
        assert np.array_equal(t.cpu().numpy().view(expect.dtype), expect)
