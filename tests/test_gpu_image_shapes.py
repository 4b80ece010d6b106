"""Device encodes at the sizes where the launch shape changes or a unit of the
bulk-copy kernel crosses block rows: around the block counts that pick the
register-loading grid or the bulk-copy kernel, rows narrower than a stage,
one block wider than a stage, padded strides.  Bit-exact with the oracle."""
import numpy as np
import pytest

import goofy_gb300 as g
import oracle
from goofy_gb300 import workloads

pytestmark = pytest.mark.gpu

# (width, height, extra stride bytes): blocks = width / 4 * height / 4
SIZES = [
    (564, 564, 0), (568, 564, 16),       # 19,881 and 20,022 blocks
    (124, 4000, 0), (128, 4000, 16),     # 31 and 32 blocks a row
    (3192, 3004, 16), (3200, 3004, 0),   # 599,298 and 600,800 blocks
    (4092, 2400, 32), (4100, 2400, 0),   # one block less / more than a stage a row
    (1020, 10000, 0), (1028, 10000, 0),  # 255 and 257 blocks a row
    (4, 40000, 0), (40000, 4, 16),       # one block a row, one row
]


def _check(cuda, img, w, h, stride, want):
    stream = cuda.cuda.current_stream().cuda_stream
    src = cuda.from_numpy(img.reshape(-1)).cuda()
    n = g.out_size(w, h)
    for codec in (g.CODEC_BC1, g.CODEC_ETC1S):
        dst = cuda.full((n + 64,), 0xA5, dtype=cuda.uint8, device="cuda")
        assert g.compress_device(codec, dst, src, w, h, stride, stream) == g.OK, g.last_error()
        got = dst.cpu().numpy()
        np.testing.assert_array_equal(got[:n], want[codec])
        assert (got[n:] == 0xA5).all()
    both = cuda.full((2 * n + 64,), 0xA5, dtype=cuda.uint8, device="cuda")
    assert g.compress_both_device(both.data_ptr(), both.data_ptr() + n, src, w, h, stride, stream) == g.OK
    got = both.cpu().numpy()
    np.testing.assert_array_equal(got[:n], want[0])
    np.testing.assert_array_equal(got[n:2 * n], want[1])
    assert (got[2 * n:] == 0xA5).all()
    assert g.pipeline_timeouts() == 0


def _image(w, h, pad):
    img = np.zeros((h, 4 * w + pad), np.uint8)
    img[:, :4 * w] = workloads.scene(w, h, seed=w + h)
    return img, 4 * w + pad, [oracle.encode(c, img, w, h, 4 * w + pad) for c in (g.CODEC_BC1, g.CODEC_ETC1S)]


@pytest.mark.parametrize("w,h,pad", SIZES)
def test_image_shapes_default_tile(cuda, w, h, pad):
    img, stride, want = _image(w, h, pad)
    _check(cuda, img, w, h, stride, want)


@pytest.mark.parametrize("threads", [128, 256, 512])
@pytest.mark.parametrize("bpt", [1, 2])
def test_bulk_copy_tiles_on_ragged_rows(cuda, threads, bpt):
    w, h, pad = 3308, 3012, 48  # 827 blocks a row: units start and end inside rows
    img, stride, want = _image(w, h, pad)
    try:
        for codec in (g.CODEC_BC1, g.CODEC_ETC1S, g.CODEC_BOTH):
            assert g.set_tile(codec, threads, bpt, 2) == g.OK
        _check(cuda, img, w, h, stride, want)
    finally:
        g.reset_tiles()


@pytest.mark.parametrize("w,h", [(564, 564), (568, 564), (124, 4000), (128, 4000), (1028, 2412), (3204, 3004),
                                 (1020, 10000), (16384, 148)])
@pytest.mark.parametrize("offset,pad", [(4, 0), (8, 4), (12, 8), (0, 12), (4, 20)])
def test_word_aligned_rows(cuda, w, h, offset, pad):
    """Rows that start 4, 8 or 12 bytes past a 16-byte boundary, the same for
    every row (pad % 16 == 0) or changing from row to row."""
    rng = np.random.default_rng(w + h)
    stride = 4 * w + pad
    img = np.zeros((h, stride), np.uint8)
    img[:, :4 * w] = workloads.scene(w, h, seed=w + offset)
    img[:, 4 * w:] = rng.integers(0, 256, (h, pad), np.uint8)
    want = [oracle.encode(c, img, w, h, stride) for c in (g.CODEC_BC1, g.CODEC_ETC1S)]
    raw = cuda.empty(h * stride + 64, dtype=cuda.uint8, device="cuda").random_(0, 256)
    src = raw[offset:offset + h * stride]
    src.copy_(cuda.from_numpy(img.reshape(-1)).cuda())
    stream = cuda.cuda.current_stream().cuda_stream
    n = g.out_size(w, h)
    for codec in (g.CODEC_BC1, g.CODEC_ETC1S):
        dst = cuda.full((n + 64,), 0xA5, dtype=cuda.uint8, device="cuda")
        assert g.compress_device(codec, dst, src, w, h, stride, stream) == g.OK, g.last_error()
        got = dst.cpu().numpy()
        np.testing.assert_array_equal(got[:n], want[codec])
        assert (got[n:] == 0xA5).all()
    both = cuda.zeros(2 * n, dtype=cuda.uint8, device="cuda")
    assert g.compress_both_device(both.data_ptr(), both.data_ptr() + n, src, w, h, stride, stream) == g.OK
    got = both.cpu().numpy()
    np.testing.assert_array_equal(got[:n], want[0])
    np.testing.assert_array_equal(got[n:], want[1])
    assert g.pipeline_timeouts() == 0
