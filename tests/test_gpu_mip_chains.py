"""Square mip chains around the sizes that one launch makes whole (512, 1024
and 2048): every level equals the host chain bit for bit, nothing else of the
arena is written, also behind another launch in the stream."""
import numpy as np
import pytest

import goofy_gb300 as g
from goofy_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [256, 512, 1024, 2048, 4096])
@pytest.mark.parametrize("offset,pad", [(0, 0), (16, 48), (4, 12)])
def test_square_chains(cuda, n, offset, pad):
    img = workloads.scene(n, n, n + offset)
    rows = np.zeros((n, 4 * n + pad), np.uint8)
    rows[:, :4 * n] = img
    raw = cuda.zeros(rows.size + 64, dtype=cuda.uint8, device="cuda")
    src = raw[offset:offset + rows.size]
    src.copy_(cuda.from_numpy(rows.reshape(-1)).cuda())
    size = g.lib().goofy_gpu_mip_arena_bytes(n, n)
    arena = cuda.full((size + 512,), 0x5A, dtype=cuda.uint8, device="cuda")
    base = arena.data_ptr() + (-arena.data_ptr()) % 256
    stream = cuda.cuda.current_stream().cuda_stream
    for _ in range(3):
        levels = g.generate_mips(src, n, n, 4 * n + pad, base, size, stream)
    assert [(lw, lh) for _, lw, lh, _ in levels] == workloads.mip_chain(n, n)
    flat, first = arena.cpu().numpy(), base - arena.data_ptr()
    written = np.zeros(flat.size, bool)
    cur, cw, ch = img, n, n
    for ptr, lw, lh, stride in levels[1:]:
        cur, cw, ch = workloads.downsample(cur, cw, ch)
        at = first + ptr - base
        np.testing.assert_array_equal(flat[at:at + stride * lh].reshape(lh, stride)[:, :4 * lw], cur[:, :4 * lw])
        written[at:at + stride * lh].reshape(lh, stride)[:, :4 * lw] = True
    assert (flat[~written] == 0x5A).all()
