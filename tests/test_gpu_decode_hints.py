"""Device codestreams at and away from the decoder's constant-bit-rate split,
and with and without vertical prediction, in long runs with several frames in
flight: every frame's result is its own, whatever the frames before it left
behind."""
import numpy as np
import pytest

import jxs_synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flight", [1, 3])
def test_long_runs(gpu, oracle, flight):
    torch = pytest.importorskip("torch")
    w, h, fmt, d = 256, 64, S.FMT_YUV422, 8
    planes = S.frame(w, h, d, fmt, seed=3)
    streams, wants = [], []
    for bpp, vpred in ((9, 0), (7, 0), (9, 1)):
        p = oracle.make_params(w, h, d, fmt, bpp, 1, 2, 5, slice_height=16, vpred=vpred)
        err, bs = oracle.oracle_encode(p, planes)[:2]
        assert err == 0
        err, want = oracle.oracle_decode(bs)
        assert err == 0
        streams.append(bs)
        wants.append(want)
    dec = gpu.Decoder(streams[0])
    heads = [b.tobytes()[:b.tobytes().index(b"\xff\x20\x00\x04")] for b in streams]
    same_header = [i for i, x in enumerate(heads) if x[:12] + x[16:] == heads[0][:12] + heads[0][16:]]  # all but Lcod
    assert 1 in same_header
    dev = [torch.from_numpy(b).cuda() for b in streams]
    # a frame away from the split, then longer runs at it than precincts are located first for, and cut ones
    order = [0] * 3 + [1] + [0] * 20 + [1] * 5 + [0] * 40 + [1, 0, 1, 0] + [0] * 70
    cuts = {30, 31, 77}
    if 2 in same_header:
        order += [2] + [0] * 5
    bufs = [[torch.zeros(x.shape, dtype=torch.uint8, device="cuda") for x in wants[0]] for _ in range(flight)]
    torch.cuda.synchronize()
    for at in range(0, len(order), flight):
        now = list(enumerate(order[at:at + flight]))
        for i, k in now:
            cut = 40 if at + i in cuts else 0
            assert dec.send(dev[k].data_ptr(), [(t.data_ptr(), t.shape[1]) for t in bufs[i]], bs_size=len(streams[k]) - cut) == 0
        for i, k in now:
            r, _ = dec.get()
            assert (r != 0) == (at + i in cuts)
            if r == 0:
                assert all(np.array_equal(t.cpu().numpy(), x) for t, x in zip(bufs[i], wants[k]))
            for t in bufs[i]:
                t.zero_()
        torch.cuda.synchronize()
    dec.close()
