"""Device-resident codestreams whose slices are not where the decoder's
constant-bit-rate split puts them: every block finds its own precinct from
that split, so such a frame is decoded again with its precincts located
first, alone and between ordinary frames."""
import numpy as np
import pytest

import jxs_synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,fmt,d,v,sl,signs,vpred", [(256, 64, S.FMT_YUV422, 8, 2, 16, 0, 0), (300, 70, S.FMT_YUV444, 10, 1, 8, 2, 0),
                                                       (320, 50, S.FMT_YUV422, 12, 2, 16, 0, 2), (260, 33, S.FMT_PACKED_RGB, 8, 0, 4, 0, 0)])
def test_slices_elsewhere(gpu, oracle, w, h, fmt, d, v, sl, signs, vpred):
    torch = pytest.importorskip("torch")
    planes = S.frame(w, h, d, fmt, seed=3)
    streams, wants = [], []
    for bpp in (9, 7):
        p = oracle.make_params(w, h, d, fmt, bpp, 1, v, 5, slice_height=sl, signs=signs, vpred=vpred)
        err, bs = oracle.oracle_encode(p, planes)[:2]
        assert err == 0
        err, want = oracle.oracle_decode(bs)
        assert err == 0
        streams.append(bs)
        wants.append(want)
    dec = gpu.Decoder(streams[0])  # its split; the second codestream differs in Lcod only
    dev = [torch.from_numpy(b).cuda() for b in streams]
    dt = torch.uint8 if d <= 8 else torch.int16
    # a cut codestream fails, and does not change how the next ones are decoded
    for k, cut in ((0, 0), (1, 0), (0, 0), (0, 40), (1, 0), (1, 31), (0, 0)):
        outs = [torch.zeros(p.shape, dtype=dt, device="cuda") for p in wants[k]]
        torch.cuda.synchronize()
        assert dec.send(dev[k].data_ptr(), [(t.data_ptr(), t.shape[1]) for t in outs], bs_size=len(streams[k]) - cut) == 0
        r, _ = dec.get()
        if cut:
            assert r in (gpu.E_DEC_TOO_SHORT, gpu.E_DEC_INVALID_BITSTREAM)
        else:
            assert r == 0
            assert all(np.array_equal(t.cpu().numpy().view(p.dtype), p) for t, p in zip(outs, wants[k]))
    dec.close()
