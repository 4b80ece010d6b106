"""The quality kernels around the sizes from which large images take the
bulk-copy ring (580,000 blocks; 2,500,000 for synchronous calls and
word-aligned rows; 256 blocks a row): the sums equal those of the decoded
image (the decoder has its own tests against the oracle)."""
import pytest

import goofy_gb300 as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,offset,pad", [
    (3200, 2896, 0, 0), (3200, 2900, 0, 16), (3204, 2900, 8, 4), (4004, 4004, 0, 0), (4000, 4000, 0, 16), (4004, 4004, 12, 4), (1020, 16000, 0, 0),
    (1024, 16000, 0, 16), (6324, 6324, 0, 0), (6324, 6324, 8, 4), (6332, 6328, 0, 16), (6332, 6328, 4, 8),
    (1028, 40000, 12, 12),
])
@pytest.mark.parametrize("codec", [0, 1])
def test_sums_of_large_images(cuda, codec, w, h, offset, pad):
    gen = cuda.Generator(device="cuda").manual_seed(w + h + codec)
    stride, k = 4 * w + pad, w * h // 2
    raw = cuda.randint(0, 256, (h * stride + 64,), dtype=cuda.uint8, device="cuda", generator=gen)
    src = raw[offset:offset + h * stride]
    blocks = cuda.empty(k, dtype=cuda.uint8, device="cuda")
    assert g.compress_device(codec, blocks, src, w, h, stride) == g.OK, g.last_error()
    cuda.cuda.synchronize()
    odd = cuda.randint(0, k // 8, (k // 80,), device="cuda", generator=gen)  # a tenth of any mode, unsupported ones too
    blocks.view(-1, 8)[odd] = cuda.randint(0, 256, (odd.numel(), 8), dtype=cuda.uint8, device="cuda", generator=gen)
    rgba = cuda.empty((h, w, 4), dtype=cuda.uint8, device="cuda")
    bad = cuda.zeros(1, dtype=cuda.int64, device="cuda")
    pitch = (4 * w + 15) // 16 * 16
    if pitch != 4 * w:
        rgba = cuda.empty((h, pitch // 4, 4), dtype=cuda.uint8, device="cuda")
    cuda.cuda.synchronize()
    assert g.decode_device(codec, rgba, pitch, blocks, w, h, bad) == g.OK, g.last_error()
    cuda.cuda.synchronize()
    d = src.view(h, stride)[:, :4 * w].reshape(h, w, 4).int() - rgba[:, :w].int()
    want = [(d[..., c] ** 2).sum().item() for c in range(4)] + [bad.item()]
    luma = ((21 * d[..., 2] + 72 * d[..., 1] + 7 * d[..., 0]).long() ** 2).sum().item()
    sums = cuda.tensor([5, 0, 0, 7, 0, 1 << 40], dtype=cuda.int64, device="cuda")  # the sums are added
    for _ in range(2):
        assert g.block_error_device(codec, blocks, src, w, h, stride, sums) == g.OK, g.last_error()
    cuda.cuda.synchronize()
    got = sums.tolist()
    assert got == [5 + 2 * want[0], 2 * want[1], 2 * want[2], 7 + 2 * want[3], 2 * want[4], (1 << 40) + 2 * luma]
    for _ in range(2):
        rc, _, five = g.psnr_rgb(codec, blocks, src, w, h, stride)
        assert rc == g.OK and five.tolist() == want
    assert g.pipeline_timeouts() == 0
