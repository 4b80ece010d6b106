"""Device encodes where the register-loading grid hands over to the bulk-copy
kernel: around the block counts that are resident at once and the largest BC1
grid, BC1 on the bulk-copy kernel with ragged rows, and sources that the
launch just before wrote (their rows are asked of L2 ahead of that launch's
end).  Bit-exact with the oracle."""
import numpy as np
import pytest

import goofy_gb300 as g
import oracle
from goofy_gb300 import workloads

pytestmark = pytest.mark.gpu

# (width, height, extra stride bytes): blocks = width / 4 * height / 4
SIZES = [
    (2048, 2128, 0), (2048, 2132, 16),   # 272,384 and 272,896 blocks
    (2048, 1824, 0), (2048, 1828, 16),   # 233,472 and 233,984
    (2500, 2560, 0), (2500, 2564, 16),   # 400,000 and 400,625
    (2048, 2432, 4), (2048, 2436, 12),   # 311,296 and 311,808, word-aligned
    (1216, 2560, 4), (1216, 2564, 20),   # 194,560 and 194,864
    (2500, 3840, 4), (2500, 3844, 4),    # 600,000 and 600,625
    (3000, 4800, 0), (3000, 4804, 16),   # 900,000 and 900,750
    (3700, 4100, 48),                    # 948,125, 925 blocks a row
    (4, 4, 0), (1024, 4, 0), (1028, 4, 0), (508, 516, 0), (120, 43000, 0),
]


@pytest.mark.parametrize("w,h,pad", SIZES)
def test_grid_and_bulk_copy_shapes(cuda, w, h, pad):
    img = np.zeros((h, 4 * w + pad), np.uint8)
    img[:, :4 * w] = workloads.scene(w, h, seed=w + h)
    want = [oracle.encode(c, img, w, h, 4 * w + pad) for c in (g.CODEC_BC1, g.CODEC_ETC1S)]
    stream = cuda.cuda.current_stream().cuda_stream
    src = cuda.from_numpy(img.reshape(-1)).cuda()
    n = g.out_size(w, h)
    for codec in (g.CODEC_BC1, g.CODEC_ETC1S):
        dst = cuda.full((n + 64,), 0xA5, dtype=cuda.uint8, device="cuda")
        assert g.compress_device(codec, dst, src, w, h, 4 * w + pad, stream) == g.OK, g.last_error()
        got = dst.cpu().numpy()
        np.testing.assert_array_equal(got[:n], want[codec])
        assert (got[n:] == 0xA5).all()
    both = cuda.full((2 * n + 64,), 0xA5, dtype=cuda.uint8, device="cuda")
    assert g.compress_both_device(both.data_ptr(), both.data_ptr() + n, src, w, h, 4 * w + pad, stream) == g.OK
    got = both.cpu().numpy()
    np.testing.assert_array_equal(got[:n], want[0])
    np.testing.assert_array_equal(got[n:2 * n], want[1])
    assert (got[2 * n:] == 0xA5).all()


@pytest.mark.parametrize("w,h", [(256, 256), (1024, 1024), (2048, 2048), (3600, 2400)])
def test_rows_written_by_the_launch_before(cuda, w, h):
    """decode -> encode -> decode -> encode through the same two buffers: each launch reads what the one before
    it in the stream wrote."""
    stream = cuda.cuda.current_stream().cuda_stream
    n = g.out_size(w, h)
    blocks = [oracle.encode(g.CODEC_BC1, workloads.scene(w, h, seed=k), w, h) for k in range(4)]
    want = []
    for b in blocks:
        px, _ = oracle.decode(g.CODEC_BC1, b, w, h)
        want.append(oracle.encode(g.CODEC_ETC1S, np.ascontiguousarray(px).reshape(h, 4 * w), w, h))
    d_blocks = [cuda.from_numpy(b).cuda() for b in blocks]
    rgba = cuda.zeros(4 * w * h, dtype=cuda.uint8, device="cuda")
    outs = [cuda.zeros(n, dtype=cuda.uint8, device="cuda") for _ in range(12)]
    bad = cuda.zeros(1, dtype=cuda.int64, device="cuda")
    cuda.cuda.synchronize()
    for k, out in enumerate(outs):
        assert g.decode_device(g.CODEC_BC1, rgba, 4 * w, d_blocks[k % 4], w, h, bad, stream) == g.OK
        assert g.compress_device(g.CODEC_ETC1S, out, rgba, w, h, 4 * w, stream) == g.OK
    for k, out in enumerate(outs):
        np.testing.assert_array_equal(out.cpu().numpy(), want[k % 4])
