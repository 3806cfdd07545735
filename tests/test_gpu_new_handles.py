"""Handles created while other work holds the device's default stream: the
first frames do not depend on anything queued behind that work."""
import ctypes
import threading
import time

import numpy as np
import pytest

import jxs_synth as S

pytestmark = pytest.mark.gpu


def leave_dirt():
    """Freed device memory that is not zero, in blocks of the sizes of a
    handle's small buffers."""
    try:
        rt = ctypes.CDLL("libcudart.so")
    except OSError:
        try:
            rt = ctypes.CDLL("/usr/local/cuda/lib64/libcudart.so")
        except OSError:
            return
    blocks = []
    for _ in range(64):
        p = ctypes.c_void_p()
        if rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(64)) == 0:
            rt.cudaMemset(p, 1, ctypes.c_size_t(64))
            blocks.append(p)
    rt.cudaDeviceSynchronize()
    for p in blocks:
        rt.cudaFree(p)


class DefaultStreamBusy:
    """Keeps the device's default stream busy, 20 ms at a time, until the end
    of the block (1 s at most)."""

    def __init__(self, torch):
        self.torch, self.stop = torch, False
        self.thread = threading.Thread(target=self.run)

    def run(self):
        end = time.perf_counter() + 1
        while not self.stop and time.perf_counter() < end:
            self.torch.cuda._sleep(int(0.02 * 1.9e9))
            time.sleep(0.015)

    def __enter__(self):
        self.thread.start()
        time.sleep(0.03)

    def __exit__(self, *a):
        self.stop = True
        self.thread.join()
        self.torch.cuda.synchronize()


def test_decoder(gpu, oracle):
    torch = pytest.importorskip("torch")
    w, h, d = 640, 64, 8
    err, bs = oracle.oracle_encode(oracle.make_params(w, h, d, S.FMT_YUV422, 5), S.frame(w, h, d, S.FMT_YUV422, seed=1))[:2]
    assert err == 0
    err, want = oracle.oracle_decode(bs)
    assert err == 0
    dev = torch.from_numpy(bs).cuda()
    outs = [torch.zeros(x.shape, dtype=torch.uint8, device="cuda") for x in want]
    gpu.Decoder(bs).close()
    leave_dirt()
    torch.cuda.synchronize()
    for _ in range(4):
        for x in outs:
            x.zero_()
        leave_dirt()
        torch.cuda.synchronize()
        got = []
        with DefaultStreamBusy(torch):
            dec = gpu.Decoder(bs)
            frame = dec.make_frame(dev.data_ptr(), [(x.data_ptr(), x.shape[1]) for x in outs], bs_size=len(bs))
            for _ in range(3):  # every slot
                assert dec.send_frame(frame) == 0
            got += [dec.get()[0] for _ in range(3)]
        assert got == [0, 0, 0]
        assert all(np.array_equal(x.cpu().numpy(), y) for x, y in zip(outs, want))
        dec.close()


def test_encoder(gpu, oracle):
    torch = pytest.importorskip("torch")
    w, h, d = 640, 64, 8
    planes = S.frame(w, h, d, S.FMT_YUV422, seed=1)
    err, want = oracle.oracle_encode(oracle.make_params(w, h, d, S.FMT_YUV422, 5), planes)[:2]
    assert err == 0
    dev = [torch.from_numpy(p).cuda() for p in planes]
    out = torch.zeros(len(want), dtype=torch.uint8, device="cuda")
    gpu.Encoder(w, h, d, S.FMT_YUV422, 5).close()
    for _ in range(4):
        out.zero_()
        leave_dirt()
        torch.cuda.synchronize()
        got = []
        with DefaultStreamBusy(torch):
            enc = gpu.Encoder(w, h, d, S.FMT_YUV422, 5)
            frame = enc.make_frame([(x.data_ptr(), x.shape[1]) for x in dev], out.data_ptr(), out.numel())
            for _ in range(3):
                assert enc.send_frame(frame) == 0
            got += [enc.get()[0] for _ in range(3)]
        assert got == [0, 0, 0]
        assert np.array_equal(out.cpu().numpy(), want)
        enc.close()
