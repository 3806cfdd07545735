"""Data positions found from the unary codes' bits: precincts with many words
of codes for each thread of the search, with less than one, with raw GCLIs in
some or all packets, without significance flags."""
import numpy as np
import pytest

import jxs_synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,fmt,d,v,bpp,sig,noise", [
    (64, 16, S.FMT_YUV422, 8, 2, 16, 1, 0), (33, 9, S.FMT_PACKED_RGB, 8, 1, 20, 0, 1),
    (1000, 32, S.FMT_YUV444, 10, 2, 2, 1, 0), (1000, 32, S.FMT_YUV444, 10, 2, 24, 1, 1),
    (4100, 18, S.FMT_YUV422, 12, 1, 4, 0, 0), (7680, 16, S.FMT_YUV444, 12, 1, 6, 1, 1),
    (7680, 16, S.FMT_YUV444, 12, 2, 3, 0, 0), (130, 40, S.FMT_YUV420, 12, 2, 9, 1, 2),
])
def test_decode_equals_oracle(gpu, oracle, w, h, fmt, d, v, bpp, sig, noise):
    torch = pytest.importorskip("torch")
    planes = S.frame(w, h, d, fmt, seed=7)
    rng = np.random.default_rng(1)
    if noise:  # a part of every line, or all of it
        for p in planes:
            n = p.shape[1] // (3 if noise == 2 else 1)
            p[:, :n] = rng.integers(0, 1 << d, (p.shape[0], n)).astype(p.dtype)
    p = oracle.make_params(w, h, d, fmt, bpp, 1, v, 5, slice_height=16, significance=sig)
    err, bs = oracle.oracle_encode(p, planes)[:2]
    assert err == 0
    err, want = oracle.oracle_decode(bs)
    assert err == 0
    dec = gpu.Decoder(bs)
    dev = torch.from_numpy(bs).cuda()
    outs = [torch.zeros(x.shape, dtype=torch.uint8 if d <= 8 else torch.int16, device="cuda") for x in want]
    torch.cuda.synchronize()
    assert dec.send(dev.data_ptr(), [(t.data_ptr(), t.shape[1]) for t in outs], bs_size=len(bs)) == 0
    r, _ = dec.get()
    assert r == 0
    assert all(np.array_equal(t.cpu().numpy().view(x.dtype), x) for t, x in zip(outs, want))
    dec.close()
