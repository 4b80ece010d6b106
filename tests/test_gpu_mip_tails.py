"""Chains whose axes reach 4 pixels at different levels (the end of such a
chain is one launch), and sources without 16-byte alignment: every level
equals the host chain bit for bit."""
import numpy as np
import pytest

import goofy_gb300 as g
from goofy_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(8, 4), (4, 16), (64, 16), (16, 64), (512, 256), (4096, 256), (256, 4096), (4096, 4),
                                 (4, 8192), (16384, 4), (8192, 8), (128, 64), (128, 128), (2048, 1024)])
@pytest.mark.parametrize("offset,pad", [(0, 0), (4, 12)])
def test_rectangular_chains(cuda, w, h, offset, pad):
    img = workloads.scene(w, h, 3 * w + h)
    rows = np.zeros((h, 4 * w + pad), np.uint8)
    rows[:, :4 * w] = img
    raw = cuda.zeros(rows.size + 64, dtype=cuda.uint8, device="cuda")
    src = raw[offset:offset + rows.size]
    src.copy_(cuda.from_numpy(rows.reshape(-1)).cuda())
    n = max(g.lib().goofy_gpu_mip_arena_bytes(w, h), 256)
    arena = cuda.full((n + 512,), 0x5A, dtype=cuda.uint8, device="cuda")
    base = arena.data_ptr() + (-arena.data_ptr()) % 256
    levels = g.generate_mips(src, w, h, 4 * w + pad, base, n, cuda.cuda.current_stream().cuda_stream)
    assert [(lw, lh) for _, lw, lh, _ in levels] == workloads.mip_chain(w, h)
    flat, first = arena.cpu().numpy(), base - arena.data_ptr()
    written = np.zeros(flat.size, bool)
    cur, cw, ch = img, w, h
    for ptr, lw, lh, stride in levels[1:]:
        cur, cw, ch = workloads.downsample(cur, cw, ch)
        at = first + ptr - base
        got = flat[at:at + stride * lh].reshape(lh, stride)
        np.testing.assert_array_equal(got[:, :4 * lw], cur[:, :4 * lw])
        written[at:at + stride * lh].reshape(lh, stride)[:, :4 * lw] = True
    assert (flat[~written] == 0x5A).all()  # nothing else was written
