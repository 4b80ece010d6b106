"""Batches of one codec and 16-byte rows against ones where a single image
differs (codec, 4-byte rows, no blocks): sizes around a warp's step of 32
blocks and a unit, by parameter table and without allocation."""
import numpy as np
import pytest

import goofy_gb300 as g
import oracle

pytestmark = pytest.mark.gpu

SIZES = [(4, 4), (128, 4), (132, 4), (4, 128), (4, 132), (252, 12), (256, 256), (260, 516), (1024, 1024), (36, 28)]


@pytest.mark.parametrize("codec", [g.CODEC_BC1, g.CODEC_ETC1S])
@pytest.mark.parametrize("odd", [None, "codec", "words", "empty"])
@pytest.mark.parametrize("at", [0, 9])
def test_one_kind_and_almost(cuda, codec, odd, at):
    images, keep, want, outs = [], [], [], []
    for k, (w, h) in enumerate(SIZES):
        kind = odd if k == at else None
        pad = 4 if kind == "words" else 16 * (k % 2)
        rows = np.zeros((h, 4 * w + pad), np.uint8)
        rows[:, :4 * w] = np.random.default_rng(k).integers(0, 256, (h, 4 * w))
        c = 1 - codec if kind == "codec" else codec
        src = cuda.from_numpy(rows.reshape(-1)).cuda()
        out = cuda.full((g.out_size(w, h) + 8,), 0xA5, dtype=cuda.uint8, device="cuda")
        keep.append(src)
        outs.append(out)
        want.append(np.full(g.out_size(w, h), 0xA5, np.uint8) if kind == "empty" else
                    oracle.encode(c, rows, w, h, 4 * w + pad))
        images.append((src.data_ptr(), out.data_ptr(), w, 0 if kind == "empty" else h, 4 * w + pad, c))
    batch = g.Batch(len(images))
    try:
        assert batch.encode(images, cuda.cuda.current_stream().cuda_stream) == g.OK
        cuda.cuda.synchronize()
    finally:
        batch.close()
    for out, ref in zip(outs, want):
        got = out.cpu().numpy()
        np.testing.assert_array_equal(got[:-8], ref)
        assert (got[-8:] == 0xA5).all()
        out.fill_(0xA5)
    assert g.batch_encode_noalloc(images, cuda.cuda.current_stream().cuda_stream) == g.OK
    for out, ref in zip(outs, want):
        np.testing.assert_array_equal(out.cpu().numpy()[:-8], ref)
