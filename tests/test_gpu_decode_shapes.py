"""The decoder at the block counts where its launch shape changes: blocks of
every mode, padded rows, the unsupported count; equal to the oracle's."""
import numpy as np
import pytest

import goofy_gb300 as g
import oracle

pytestmark = pytest.mark.gpu

# 429,680 / 430,336 / 1,249,924 / 1,251,042 blocks; one block; one row; one block a row
SIZES = [(2620, 2624), (2624, 2624), (4472, 4472), (4476, 4472), (4, 4), (4100, 4), (4, 4100)]


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("codec", [0, 1])
def test_decode_shapes(cuda, codec, w, h):
    rng = np.random.default_rng(w * 7 + h + codec)
    n = (w // 4) * (h // 4)
    blocks = rng.integers(0, 256, (n, 8), dtype=np.uint8)
    if codec == 1:  # half of them of the shape that the encoder writes
        blocks[::2, :3] &= 0xF8
        blocks[::2, 3] = (blocks[::2, 3] >> 5) * 0x24 + 2
    blocks = blocks.reshape(-1)
    want, bad = oracle.decode(codec, blocks, w, h)
    stride = 4 * w + 48
    out = cuda.full((h, stride), 0xA5, dtype=cuda.uint8, device="cuda")
    count = cuda.tensor([3], dtype=cuda.int64, device="cuda")
    assert g.decode_device(codec, out, stride, cuda.from_numpy(blocks).cuda(), w, h, count) == g.OK, g.last_error()
    got = out.cpu().numpy()
    np.testing.assert_array_equal(got[:, :4 * w], want.reshape(h, 4 * w))
    assert (got[:, 4 * w:] == 0xA5).all()
    assert int(count.item()) == 3 + bad
