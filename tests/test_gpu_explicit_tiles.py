"""Grids asked for by their shape, around the sizes at which they stop asking
L2 for their rows early (one wave of CTAs, 1,250,000 blocks): the blocks equal
those of the default tile, which has its own tests against the oracle."""
import pytest

import goofy_gb300 as g

pytestmark = pytest.mark.gpu


@pytest.fixture
def tiles():
    yield
    g.reset_tiles()


@pytest.mark.parametrize("w,h", [(2048, 1216), (2048, 1220), (2048, 1824), (2048, 1828), (2052, 2124), (4000, 5000),
                                 (4000, 5004)])
@pytest.mark.parametrize("offset,pad", [(0, 0), (4, 8)])
def test_explicit_grids_equal_the_default_tile(cuda, tiles, w, h, offset, pad):
    stride, n = 4 * w + pad, g.out_size(w, h)
    gen = cuda.Generator(device="cuda").manual_seed(w + h + pad)
    src = cuda.randint(0, 256, (h * stride + 64,), dtype=cuda.uint8, device="cuda", generator=gen)[offset:]
    want, got = (cuda.empty(2 * n, dtype=cuda.uint8, device="cuda") for _ in range(2))

    def encode(codec, out):
        out.zero_()
        cuda.cuda.synchronize()
        if codec == g.CODEC_BOTH:
            rc = g.compress_both_device(out, out[n:], src, w, h, stride)
        else:
            rc = g.compress_device(codec, out, src, w, h, stride)
        assert rc == g.OK, g.last_error()
        cuda.cuda.synchronize()

    for codec in (g.CODEC_BC1, g.CODEC_ETC1S, g.CODEC_BOTH):
        g.reset_tiles()
        encode(codec, want)
        for threads in (128, 256, 512):
            for bpt in (1, 2, 4)[:2 if codec == g.CODEC_BOTH else 3]:
                assert g.set_tile(codec, threads, bpt, 0) == g.OK
                encode(codec, got)
                assert cuda.equal(got, want), (codec, threads, bpt)
