"""Codestreams do not depend on what the working memory held before: bands
whose width is not a multiple of four coefficients, at every horizontal level
and in every layout of lanes, on memory full of another frame's data."""
import numpy as np
import pytest

import jxs_synth as S

pytestmark = pytest.mark.gpu

# (w, h, depth, format, bpp, V, H, signs, prediction); the horizontal-only
# levels start from widths 169, 480, 130, 83, 960, 45, 250, 1 and so on
SHAPES = [(338, 106, 12, S.FMT_YUV420, 11, 1, 5, 2, 0), (1920, 32, 8, S.FMT_YUV422, 5, 2, 5, 0, 0), (130, 24, 8, S.FMT_YUV444, 20, 0, 5, 0, 0),
          (330, 40, 10, S.FMT_YUV444, 12, 2, 4, 1, 0), (3840, 16, 10, S.FMT_YUV422, 3, 2, 5, 0, 0), (178, 33, 14, S.FMT_PACKED_RGB, 20, 2, 3, 0, 0),
          (500, 48, 8, S.FMT_YUV422, 9, 1, 5, 0, 1), (777, 20, 12, S.FMT_YUV444, 9, 1, 2, 2, 2), (1000, 16, 8, S.FMT_PACKED_RGB, 9, 0, 4, 0, 0)]


def oracle_bytes(oracle, w, h, d, fmt, bpp, v, hh, signs, vpred):
    planes = S.frame(w, h, d, fmt, seed=w + h)
    err, want = oracle.oracle_encode(oracle.make_params(w, h, d, fmt, bpp, 1, v, hh, signs=signs, vpred=vpred), planes)[:2]
    assert err == 0
    return planes, want


def encoder(gpu, w, h, d, fmt, bpp, v, hh, signs, vpred):
    return gpu.Encoder(w, h, d, fmt, bpp, 1, v, hh, coding_signs_handling=signs, coding_vertical_prediction_mode=vpred)


def test_batches_in_the_memory_of_others(gpu, oracle):
    """One arena, just large enough for a frame of noise, whose working set the
    other frames take over one after another."""
    w, h, d = 1500, 360, 14
    rng = np.random.default_rng(1)
    noise = [rng.integers(0, 1 << d, (h, w)).astype(np.uint16) for _ in range(3)]
    big = gpu.Encoder(w, h, d, S.FMT_YUV444, 20, 1, 1, 5, coding_signs_handling=2)
    want_big = big.encode(noise)
    out_big = np.zeros(big.frame_bytes + 64, np.uint8)
    for mb in range(8, 400, 4):
        batch = gpu.Batch(mb << 20)
        if batch.encode([big], [noise], [out_big]) == 0:
            break
        batch.close()
    assert batch.wait()[0] == 0 and np.array_equal(out_big[:len(want_big)], want_big)
    wrong = []
    for shape in SHAPES:
        planes, want = oracle_bytes(oracle, *shape)
        enc = encoder(gpu, *shape)
        out = np.zeros(enc.frame_bytes + 64, np.uint8)
        assert batch.encode([enc], [planes], [out]) == 0
        if batch.wait()[0] != 0 or not np.array_equal(out[:len(want)], want):
            wrong.append(shape)
        enc.close()
        assert batch.encode([big], [noise], [out_big]) == 0  # takes the memory back
        assert batch.wait()[0] == 0 and np.array_equal(out_big[:len(want_big)], want_big)
    batch.close()
    big.close()
    assert not wrong
