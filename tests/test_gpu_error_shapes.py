"""The quality kernels at the sizes where their launch shape changes, with
vector- and word-aligned sources, ETC1 blocks of every mode and several
threads: the sums equal the oracle's."""
import threading

import numpy as np
import pytest

import goofy_gb300 as g
import oracle
from goofy_gb300 import workloads

pytestmark = pytest.mark.gpu

# (width, height, source offset, extra stride bytes)
SHAPES = [
    (4, 4, 0, 0), (564, 564, 0, 0), (568, 564, 0, 16), (124, 4000, 4, 0), (128, 4000, 0, 0), (128, 4000, 8, 4),
    (1020, 1020, 0, 12), (3192, 3004, 0, 0), (3200, 3004, 0, 16), (3200, 3004, 12, 0), (1020, 10000, 0, 0),
    (1028, 10000, 4, 8),
]


def _want(codec, blocks, img, w, h):
    px, bad = oracle.decode(codec, blocks, w, h)
    d = img.reshape(h, w, 4).astype(np.int64) - px.reshape(h, w, 4).astype(np.int64)
    luma = int(((21 * d[..., 2] + 72 * d[..., 1] + 7 * d[..., 0]) ** 2).sum())
    return [int((d[..., c] ** 2).sum()) for c in range(4)] + [bad, luma]


def _device_source(cuda, img, offset, pad):
    h, row = img.shape
    rows = np.full((h, row + pad), 77, np.uint8)
    rows[:, :row] = img
    raw = cuda.zeros(h * (row + pad) + 64, dtype=cuda.uint8, device="cuda")
    src = raw[offset:offset + h * (row + pad)]
    src.copy_(cuda.from_numpy(rows.reshape(-1)).cuda())
    return src


@pytest.mark.parametrize("w,h,offset,pad", SHAPES)
@pytest.mark.parametrize("codec", [0, 1])
def test_sums_at_every_shape(cuda, codec, w, h, offset, pad):
    rng = np.random.default_rng(w + h + codec)
    img = np.ascontiguousarray(workloads.scene(w, h, seed=w)[:, :4 * w])
    img.reshape(h, w, 4)[..., 3] = rng.integers(0, 256, (h, w))
    blocks = oracle.encode(codec, img, w, h)
    odd = rng.integers(0, blocks.size // 8, max(1, blocks.size // 80))  # a tenth of any mode, unsupported ones too
    blocks.reshape(-1, 8)[odd] = rng.integers(0, 256, (odd.size, 8))
    want = _want(codec, blocks, img, w, h)
    src = _device_source(cuda, img, offset, pad)
    blk = cuda.from_numpy(blocks).cuda()
    sums = cuda.tensor([5, 0, 0, 7, 0, 1 << 40], dtype=cuda.int64, device="cuda")  # the sums are added
    for _ in range(2):
        assert g.block_error_device(codec, blk, src, w, h, 4 * w + pad, sums) == g.OK, g.last_error()
    got = sums.cpu().numpy().tolist()
    assert got == [5 + 2 * want[0], 2 * want[1], 2 * want[2], 7 + 2 * want[3], 2 * want[4], (1 << 40) + 2 * want[5]]
    for _ in range(2):  # the synchronous form starts from zero each time
        rc, psnr, five = g.psnr_rgb(codec, blk, src, w, h, 4 * w + pad)
        assert rc == g.OK and five.tolist() == want[:5] and psnr == oracle.psnr_rgb(five, w, h)
    assert g.mse_psnr(codec, blk, src, w, h, 4 * w + pad)["mse_y"] == pytest.approx(want[5] / 1e4 / (w * h), rel=1e-12)
    assert g.pipeline_timeouts() == 0


def test_concurrent_callers_get_their_own_sums(cuda):
    """Four threads measure different images at once; every answer is its own image's."""
    jobs = []
    for k, (w, h) in enumerate(((256, 256), (1024, 512), (2048, 1024), (640, 640))):
        img = np.ascontiguousarray(workloads.scene(w, h, seed=k)[:, :4 * w])
        blocks = oracle.encode(k % 2, img, w, h)
        jobs.append((k % 2, cuda.from_numpy(blocks).cuda(), _device_source(cuda, img, 0, 0), w, h,
                     _want(k % 2, blocks, img, w, h)[:5]))
    cuda.cuda.synchronize()
    wrong = []

    def work(codec, blk, src, w, h, want):
        for _ in range(50):
            rc, _, five = g.psnr_rgb(codec, blk, src, w, h, 4 * w)
            if rc != g.OK or five.tolist() != want:
                wrong.append((w, h, rc, five.tolist(), want))

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:3]
