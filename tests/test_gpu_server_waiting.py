"""Batched serving loop: a request for which a lane is idle starts at once."""
import time

import numpy as np
import pytest

import jxs_synth as S

pytestmark = pytest.mark.gpu
GB = 1 << 30


def stream(gpu, torch, w, h, d, bpp):
    enc = gpu.Encoder(w, h, d, S.FMT_YUV422, bpp)
    planes = [torch.from_numpy(p.view(np.int16) if p.dtype == np.uint16 else p).cuda() for p in S.frame(w, h, d, S.FMT_YUV422, seed=3)]
    out = torch.zeros(enc.frame_bytes, dtype=torch.uint8, device="cuda")
    return enc, planes, [(t.data_ptr(), t.shape[1]) for t in planes], out


def spin(us):
    t = time.perf_counter() + us * 1e-6
    while time.perf_counter() < t:
        pass


def drain(server, n):
    got, t0 = [], time.time()
    while len(got) < n:
        got.extend(server.poll())
        assert time.time() - t0 < 60
    assert all(d[2] == 0 for d in got)
    return got


def test_small_frame_beside_a_large_one(gpu):
    """Of two lanes one encodes a 4K frame: a small frame does not wait for
    the other.  The least wait of 60, so that a busy host does not matter."""
    torch = pytest.importorskip("torch")
    big, small = stream(gpu, torch, 3840, 2160, 10, 3), stream(gpu, torch, 256, 64, 8, 5)
    server = gpu.Server(2 * GB, gpu.SERVER_BATCHED, lanes=2, max_batch=16)
    ids = [server.add_encoder(x[0]) for x in (big, small)]
    torch.cuda.synchronize()
    waits = []
    for _ in range(60):
        assert server.submit(ids[0], 0, big[2], big[3].data_ptr()) == 0
        spin(40)
        assert server.submit(ids[1], 1, small[2], small[3].data_ptr()) == 0
        waits += [start - arrive for tag, _, _, arrive, start, _ in drain(server, 2) if tag == 1]
        spin(200)
    server.close()
    assert min(waits) < 20000


def test_two_small_frames_on_three_idle_lanes(gpu):
    torch = pytest.importorskip("torch")
    streams = [stream(gpu, torch, 256, 64, 8, 5) for _ in range(2)]
    server = gpu.Server(2 * GB, gpu.SERVER_BATCHED, lanes=3, max_batch=16)
    ids = [server.add_encoder(x[0]) for x in streams]
    torch.cuda.synchronize()
    for _ in range(100):
        for i, x in enumerate(streams):
            assert server.submit(ids[i], i, x[2], x[3].data_ptr()) == 0
        drain(server, 2)
        spin(400)
    st = server.stats()
    server.close()
    assert st["batches"] == st["batched_frames"] == 200
