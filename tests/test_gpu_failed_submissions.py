"""A submission that fails half way (a page-locked plane whose rows lie closer
together than they are long, which the copy call refuses) hands the caller's
buffers back: nothing that it had queued is still reading or writing them when
the error arrives, and the handle's next frames are right."""
import numpy as np
import pytest

import jxs_synth as S

pytestmark = pytest.mark.gpu

W, H, D, BPP = 3840, 2160, 10, 3


def pinned(torch, a):
    return torch.from_numpy(a.view(np.int16)).pin_memory()


def narrow_last_plane(frame, n, w, h):
    """The last plane's rows one sample too close together; the plane itself
    is large enough by the caller's account."""
    frame.image.stride[n - 1] = w - 1
    frame.image.alloc_size[n - 1] = 2 * w * h
    return frame


def test_decode(gpu, oracle):
    torch = pytest.importorskip("torch")
    planes = S.frame(W, H, D, S.FMT_YUV422, seed=1)
    enc = gpu.Encoder(W, H, D, S.FMT_YUV422, BPP)
    bs = enc.encode(planes)
    enc.close()
    dec = gpu.Decoder(bs)
    want = dec.decode(bs)
    stream = torch.cuda.Stream()
    dec.set_stream(stream.cuda_stream)
    outs = [pinned(torch, np.zeros_like(p)) for p in want]
    ptrs = [(t.data_ptr(), t.shape[1]) for t in outs]
    bad = narrow_last_plane(dec.make_frame(bs, ptrs), 3, W // 2, H)
    good = dec.make_frame(bs, ptrs)
    for _ in range(5):
        # the codestream from pageable memory: its copy is under way before
        # the rest of the frame is queued
        assert dec.send_frame(bad) == 0
        r, _ = dec.get()
        assert r != 0
        assert stream.query(), "the failed frame's work still runs"
        for t in outs:
            t.zero_()
        assert dec.send_frame(good) == 0
        r, _ = dec.get()
        assert r == 0
        assert all(np.array_equal(t.numpy().view(p.dtype), p) for t, p in zip(outs, want))
    dec.close()


def test_encode(gpu, oracle):
    torch = pytest.importorskip("torch")
    planes = S.frame(W, H, D, S.FMT_YUV422, seed=2)
    enc = gpu.Encoder(W, H, D, S.FMT_YUV422, BPP)
    want = enc.encode(planes)
    stream = torch.cuda.Stream()
    enc.set_stream(stream.cuda_stream)
    ins = [pinned(torch, p) for p in planes]
    out = np.ones(enc.frame_bytes + 64, np.uint8)
    ptrs = [(t.data_ptr(), t.shape[1]) for t in ins]
    bad = narrow_last_plane(enc.make_frame(ptrs, out), 3, W // 2, H)
    pageable = [p.copy() for p in planes]
    good = enc.make_frame(pageable, out)
    for _ in range(5):
        assert enc.send_frame(bad) == 0
        r, _ = enc.get()
        assert r != 0
        assert stream.query(), "the failed frame's work still runs"
        out[:] = 1
        assert enc.send_frame(good) == 0
        r, f = enc.get()
        assert r == 0 and np.array_equal(out[:f.bitstream.used_size], want)
    enc.close()
