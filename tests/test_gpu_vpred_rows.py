"""Vertical prediction with a cluster of blocks per slice: slices of fewer,
as many and more rows than blocks, a short last slice, one slice for the whole
picture, and codestreams that end within a slice between good ones."""
import numpy as np
import pytest

import jxs_synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,fmt,d,v,sl,mode,signs", [
    (300, 50, S.FMT_YUV422, 10, 2, 16, 1, 0), (300, 61, S.FMT_YUV444, 8, 1, 16, 2, 2), (200, 97, S.FMT_YUV422, 8, 0, 32, 1, 1),
    (320, 200, S.FMT_YUV420, 8, 1, 200, 2, 0), (256, 36, S.FMT_YUV422, 12, 2, 12, 1, 0), (129, 24, S.FMT_YUV444, 10, 2, 4, 2, 0),
    (1024, 1100, S.FMT_YUV422, 8, 1, 8, 1, 0),
])
def test_rows_of_a_slice(gpu, oracle, w, h, fmt, d, v, sl, mode, signs):
    torch = pytest.importorskip("torch")
    p = oracle.make_params(w, h, d, fmt, 8, 1, v, 5, slice_height=sl, vpred=mode, signs=signs)
    err, bs = oracle.oracle_encode(p, S.frame(w, h, d, fmt, seed=11))[:2]
    assert err == 0
    err, want = oracle.oracle_decode(bs)
    assert err == 0
    dec = gpu.Decoder(bs)
    dev = torch.from_numpy(bs).cuda()
    outs = [torch.zeros(x.shape, dtype=torch.uint8 if d <= 8 else torch.int16, device="cuda") for x in want]
    for cut in (0, len(bs) // 3, 0, 25, 0):
        for t in outs:
            t.zero_()
        torch.cuda.synchronize()
        assert dec.send(dev.data_ptr(), [(t.data_ptr(), t.shape[1]) for t in outs], bs_size=len(bs) - cut) == 0
        r, _ = dec.get()
        assert (r != 0) == (cut != 0)
        if not cut:
            assert all(np.array_equal(t.cpu().numpy().view(x.dtype), x) for t, x in zip(outs, want))
    dec.close()
