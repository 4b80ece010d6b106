"""The work that is timed: what a user of this library has it do, through its public entry points.

* ``listed()``           named cases, from the smallest call to the largest
* ``draw(rng)``          one more case of the same ranges
* ``prepare(case, seed)`` what a program holds before the call: images on the GPU (or in host memory where the
                         call takes host memory), output buffers, batch objects and descriptor arrays
* ``run(state)``         one pass; returns the whole outputs
* ``work(case)``         bytes that a pass cannot do without
* ``exact(case, seed)``  the floating-point results in 64 bits, by plain torch

The images are made on the GPU from the seed: a colour gradient, four octaves of smooth noise and rectangles of one
colour, as a photograph or a painted texture has them, or the four degenerate quarters (noise, one colour a block, two
colours a block, grey noise with random alpha).
"""
import math
import sys

import numpy as np
import torch

import goofy_gb300 as g
from goofy_gb300 import workloads

BC1, ETC1S = "bc1", "etc1s"


# ---- the cases -------------------------------------------------------------------------------------------------

def listed():
    return [
        # The smallest host call: the drop-in on the 256x256 plain image, from and to ordinary (pageable) memory.
        # A tool that encodes one small texture at a time waits for each: latency counts, not bandwidth.
        {"name": "dropin_bc1_256", "kind": "dropin", "codec": BC1, "width": 256, "height": 256},
        # The same call on a full-size material texture, where the rows cross the host link.
        {"name": "dropin_etc1s_2048", "kind": "dropin", "codec": ETC1S, "width": 2048, "height": 2048},
        # A streaming thread's upload of two dozen virtual-texture tiles through the entry point that allocates
        # nothing: the smallest device work that a frame does.
        {"name": "stream_24_tiles_128", "kind": "stream", "count": 24, "width": 128, "height": 128},
        # An image of screen size in both formats, one call after the other, as the harness encodes each image.
        {"name": "pair_1920x1080", "kind": "pair", "width": 1920, "height": 1080},
        # The stress image of the benchmark in the more costly codec.
        {"name": "etc1s_4096_stress", "kind": "single", "codec": ETC1S, "width": 4096, "height": 4096, "stress": True},
        # The largest single image of the benchmark.
        {"name": "bc1_8192", "kind": "single", "codec": BC1, "width": 8192, "height": 8192, "stress": False},
        # Both formats of a material texture from one read of it (a pipeline that ships both).
        {"name": "both_2048", "kind": "both", "width": 2048, "height": 2048},
        # A part of a larger atlas at an odd pixel offset: rows that are only 4-byte aligned, a ragged size.
        {"name": "crop_etc1s_1996x1532", "kind": "crop", "codec": ETC1S, "width": 1996, "height": 1532, "offset": 3,
         "pad": 101},
        # The mixed batch of the benchmark: 1000 textures of 64..2048 pixels, a fifth with mip chains, both codecs.
        {"name": "batch_1000_textures", "kind": "batch", "count": 1000, "first": 0},
        # The import of one texture: its mip chain made on the device, all levels encoded in one batch call.
        {"name": "import_2048_chain", "kind": "import", "codec": BC1, "width": 2048, "height": 2048, "pad": 0},
        # Decoding an image of screen size for a viewer or a comparison.
        {"name": "decode_etc1s_3840x2160", "kind": "decode", "codec": ETC1S, "width": 3840, "height": 2160},
        # The quality record of one encoded image (the harness's getMsePsnr), read back by the caller.
        {"name": "quality_bc1_4096", "kind": "quality", "codec": BC1, "width": 4096, "height": 4096},
    ]


def _spread(rng, lo, hi, step):
    """A multiple of `step` in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(max(round(v / step) * step, lo), hi))


def _size(rng, lo, hi, step, most=1 << 40, least=0):
    for _ in range(1000):
        w, h = _spread(rng, lo, hi, step), _spread(rng, lo, hi, 4)
        if least <= w * h <= most:
            return w, h
    raise ValueError("no size in range")


def draw(rng):
    kind = rng.choice(["dropin", "stream", "pair", "single", "single", "both", "crop", "batch", "import", "decode",
                       "quality"])
    codec = rng.choice([BC1, ETC1S])
    if kind == "dropin":  # the reference's own size rule: widths a multiple of 16
        w, h = _size(rng, 64, 3072, 16, most=2048 * 2048)
        return {"kind": kind, "codec": codec, "width": w, "height": h}
    if kind == "stream":
        w, h = _size(rng, 32, 512, 4)
        return {"kind": kind, "count": rng.randint(2, 256) if w * h <= 128 * 128 else rng.randint(2, 64),
                "width": w, "height": h}
    if kind == "pair":
        w, h = _size(rng, 256, 4096, 4)
        return {"kind": kind, "width": w, "height": h}
    if kind == "single":  # large enough that a pass is more than the call itself
        w, h = _size(rng, 512, 8192, 4, least=2048 * 1536)
        return {"kind": kind, "codec": codec, "width": w, "height": h, "stress": rng.random() < 0.25}
    if kind == "both":
        w, h = _size(rng, 512, 8192, 4, least=2048 * 1536)
        return {"kind": kind, "width": w, "height": h}
    if kind == "crop":
        w, h = _size(rng, 512, 4096, 4, least=1024 * 1024)
        return {"kind": kind, "codec": codec, "width": w, "height": h, "offset": rng.randint(1, 3),
                "pad": rng.randint(4, 515)}
    if kind == "batch":
        return {"kind": kind, "count": _spread(rng, 8, 1000, 1), "first": rng.randint(0, 5000)}
    if kind == "import":
        return {"kind": kind, "codec": codec, "width": 1 << rng.randint(8, 12), "height": 1 << rng.randint(8, 12),
                "pad": 4 * rng.randint(0, 64)}  # pixels between the rows of a pitched source
    w, h = _size(rng, 1024, 8192, 4, least=2560 * 2048 if kind == "decode" else 0)  # decode, quality
    return {"kind": kind, "codec": codec, "width": w, "height": h}


# ---- images ----------------------------------------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _scene(gen, h, w):
    """(h, w, 4) uint8: gradient, four octaves of smooth noise, rectangles; alpha 255."""
    dev = "cuda"
    y = torch.linspace(0, 255, h, device=dev).view(1, h, 1)
    x = torch.linspace(0, 255, w, device=dev).view(1, 1, w)
    img = torch.cat([x.expand(1, h, w), y.expand(1, h, w), (x + y) / 2], 0).contiguous()
    scale = max(1, max(h, w) // 256)
    for period, amp in ((64 * scale, 48.0), (32 * scale, 24.0), (16 * scale, 12.0), (8, 8.0)):
        noise = torch.rand(1, 3, h // period + 2, w // period + 2, device=dev, generator=gen) * 2 - 1
        img += amp * torch.nn.functional.interpolate(noise, size=(h, w), mode="bilinear", align_corners=False)[0]
    out = torch.full((h, w, 4), 255, dtype=torch.uint8, device=dev)
    out[..., :3] = img.clamp_(0, 255).to(torch.uint8).permute(1, 2, 0)
    n = min(256, max(8, h * w // 65536))
    box = torch.rand(n, 4, generator=gen, device=dev).cpu().tolist()
    fill = torch.randint(0, 256, (n, 3), generator=gen, device=dev, dtype=torch.uint8)
    for (a, b, c, d), colour in zip(box, fill):
        y0, x0 = int(a * h), int(b * w)
        out[y0:y0 + 8 + int(c * 88), x0:x0 + 8 + int(d * 88), :3] = colour
    return out


def _stress(gen, h, w):
    """(h, w, 4) uint8: vertical quarters of noise / one colour a block / two colours a block / grey noise."""
    out = torch.randint(0, 256, (h, w, 4), dtype=torch.uint8, device="cuda", generator=gen)
    q = w // 4 // 4 * 4
    if q:
        blocks = torch.randint(0, 256, (2, h // 4, q // 4, 4), dtype=torch.uint8, device="cuda", generator=gen)
        one, two = (b.repeat_interleave(4, 0).repeat_interleave(4, 1) for b in blocks)
        out[:, q:2 * q] = one
        pick = torch.rand(h, q, 1, device="cuda", generator=gen) < 0.5
        out[:, 2 * q:3 * q] = torch.where(pick, one, two)
        out[:, 3 * q:, 1] = out[:, 3 * q:, 0]
        out[:, 3 * q:, 2] = out[:, 3 * q:, 0]
    return out


def _codec(case):
    return g.CODECS[case["codec"]]


def _out(*shape):
    return torch.zeros(shape, dtype=torch.uint8, device="cuda")


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _images(gen, sizes):
    """Device images of the given (width, height, codec): parts of one scene, back to back in one buffer with
    256-byte aligned starts, and their output buffer; (descriptor array, source buffer, output buffer)."""
    side_w, side_h = max(w for w, _, _ in sizes), max(h for _, h, _ in sizes)
    big = _scene(gen, side_h + 512, side_w + 512)
    at = torch.randint(0, 513, (len(sizes), 2), generator=gen, device="cuda").cpu().tolist()
    src_at, dst_at, src_n, dst_n = [], [], 0, 0
    for w, h, _ in sizes:
        src_at.append(src_n)
        dst_at.append(dst_n)
        src_n += (4 * w * h + 255) // 256 * 256
        dst_n += (g.out_size(w, h) + 255) // 256 * 256
    src, dst = _out(src_n), _out(dst_n)
    array = []
    for i, (w, h, codec) in enumerate(sizes):
        y, x = at[i]
        src[src_at[i]:src_at[i] + 4 * w * h].view(h, w, 4).copy_(big[y:y + h, x:x + w])
        array.append((src.data_ptr() + src_at[i], dst.data_ptr() + dst_at[i], w, h, 4 * w, codec))
    return g.images_array(array), src, dst


def _texture_sizes(case):
    """(width, height, codec) of every level of the mixed batch's textures."""
    return [(im["width"], im["height"], im["codec"])
            for im in workloads.texture_batch(case["count"], case["first"], with_pixels=False)]


def _tile_sizes(case):
    return [(case["width"], case["height"], i % 2) for i in range(case["count"])]


# ---- prepare and run -------------------------------------------------------------------------------------------

def prepare(case, seed):
    kind, gen = case["kind"], _generator(seed)
    s = {"kind": kind, "stream": _stream()}
    if kind in ("batch", "stream"):
        sizes = _texture_sizes(case) if kind == "batch" else _tile_sizes(case)
        s["images"], s["src"], s["dst"] = _images(gen, sizes)
        if kind == "batch":
            s["batch"] = g.Batch(len(sizes))
        return s
    w, h = case["width"], case["height"]
    s.update(width=w, height=h, stride=4 * w)
    blocks = g.out_size(w, h)
    if kind == "crop":  # a part of a larger image, `offset` pixels off a block boundary
        atlas = _scene(gen, h, w + case["pad"])
        s.update(codec=_codec(case), atlas=atlas, stride=4 * (w + case["pad"]), dst=_out(blocks),
                 src=atlas[:, case["offset"]:case["offset"] + w])
        return s
    src = (_stress if case.get("stress") else _scene)(gen, h, w + case.get("pad", 0))
    if kind == "dropin":
        s.update(src=src.cpu().numpy(), dst=np.zeros(blocks, np.uint8),
                 call=g.compressDXT1 if case["codec"] == BC1 else g.compressETC1)
    elif kind in ("pair", "both"):
        s.update(src=src, bc1=_out(blocks), etc1s=_out(blocks))
    elif kind == "single":
        s.update(codec=_codec(case), src=src, dst=_out(blocks))
    elif kind == "import":
        n = g.lib().goofy_gpu_mip_arena_bytes(w, h)
        arena = _out(n + 256)
        arena = arena[-arena.data_ptr() % 256:][:n]
        s["stride"] = 4 * (w + case["pad"])
        levels = g.generate_mips(src, w, h, s["stride"], arena, n, s["stream"])  # the arena's layout, always the same
        total = sum(g.out_size(lw, lh) for _, lw, lh, _ in levels)
        dst, at, array = _out(total), 0, []
        for ptr, lw, lh, stride in levels:
            array.append((ptr, dst.data_ptr() + at, lw, lh, stride, _codec(case)))
            at += g.out_size(lw, lh)
        s.update(src=src, arena=arena, arena_bytes=n, dst=dst, images=g.images_array(array),
                 batch=g.Batch(len(array)))
    else:  # decode, quality: the image's own blocks
        dst = _out(blocks)
        _ok(g.compress_device(_codec(case), dst, src, w, h, 4 * w, s["stream"]))
        s.update(codec=_codec(case), src=src, blocks=dst)
        if kind == "decode":
            s.update(rgba=_out(h, w, 4), unsupported=torch.zeros(1, dtype=torch.int64, device="cuda"))
    return s


def _ok(status):
    if status != g.OK:
        raise RuntimeError("%s %s" % (g.status_string(status), g.last_error()))


def run(s):
    kind = s["kind"]
    if kind == "batch":
        _ok(s["batch"].encode(s["images"], s["stream"]))
        return s["dst"]
    if kind == "stream":
        _ok(g.batch_encode_noalloc(s["images"], s["stream"]))
        return s["dst"]
    w, h, stride, stream = s["width"], s["height"], s["stride"], s["stream"]
    if kind == "dropin":
        _ok(s["call"](s["dst"], s["src"], w, h, stride))
        return s["dst"]
    if kind in ("single", "crop"):
        _ok(g.compress_device(s["codec"], s["dst"], s["src"], w, h, stride, stream))
        return s["dst"]
    if kind == "pair":
        _ok(g.compress_device(g.CODEC_BC1, s["bc1"], s["src"], w, h, stride, stream))
        _ok(g.compress_device(g.CODEC_ETC1S, s["etc1s"], s["src"], w, h, stride, stream))
        return s["bc1"], s["etc1s"]
    if kind == "both":
        _ok(g.compress_both_device(s["bc1"], s["etc1s"], s["src"], w, h, stride, stream))
        return s["bc1"], s["etc1s"]
    if kind == "import":
        g.generate_mips(s["src"], w, h, stride, s["arena"], s["arena_bytes"], stream)
        _ok(s["batch"].encode(s["images"], stream))
        return s["arena"], s["dst"]
    if kind == "decode":
        _ok(g.decode_device(s["codec"], s["rgba"], 4 * w, s["blocks"], w, h, s["unsupported"], stream))
        return s["rgba"], s["unsupported"]
    return g.mse_psnr(s["codec"], s["blocks"], s["src"], w, h, stride)


# ---- what a pass cannot do without -------------------------------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind in ("batch", "stream"):
        px = sum(w * h for w, h, _ in (_texture_sizes(case) if kind == "batch" else _tile_sizes(case)))
        return {"bytes": 4.5 * px, "flops": 0}
    px = case["width"] * case["height"]
    if kind == "pair":  # two independent calls, each reads the image
        return {"bytes": 9 * px, "flops": 0}
    if kind == "both":
        return {"bytes": 5 * px, "flops": 0}
    if kind == "import":  # level 0 read, the others written, the blocks of all written
        levels = sum(w * h for w, h in workloads.mip_chain(case["width"], case["height"]))
        return {"bytes": 4 * px + 4 * (levels - px) + 0.5 * levels, "flops": 0}
    return {"bytes": 4.5 * px, "flops": 0}  # dropin, single, crop, decode, quality


# ---- 64-bit values of the floating-point results -------------------------------------------------------------------

def _decode_bc1(blocks, h, w):
    """(h, w, 4) int64 of BC1 blocks (both endpoint orders)."""
    b = blocks.view(h // 4, w // 4, 8).to(torch.int64)
    c0, c1 = b[..., 0] | b[..., 1] << 8, b[..., 2] | b[..., 3] << 8

    def rgb(c):
        r, gr, bl = c >> 11 & 31, c >> 5 & 63, c & 31
        return torch.stack([r << 3 | r >> 2, gr << 2 | gr >> 4, bl << 3 | bl >> 2], -1)

    p, q, four = rgb(c0), rgb(c1), (c0 > c1)[..., None]
    pal = torch.stack([p, q, torch.where(four, (2 * p + q) // 3, (p + q) // 2),
                       torch.where(four, (p + 2 * q) // 3, 0)], -2)
    alpha = torch.full(pal.shape[:-1] + (1,), 255, dtype=torch.int64, device=pal.device)
    alpha[..., 3, 0] = torch.where(four[..., 0], 255, 0)
    pal = torch.cat([pal, alpha], -1)
    bits = b[..., 4] | b[..., 5] << 8 | b[..., 6] << 16 | b[..., 7] << 24
    idx = torch.stack([bits >> 2 * i & 3 for i in range(16)], -1)
    px = torch.gather(pal, -2, idx[..., None].expand(idx.shape + (4,)))
    return px.view(h // 4, w // 4, 4, 4, 4).permute(0, 2, 1, 3, 4).reshape(h, w, 4)


def _decode_etc1s(blocks, h, w):
    """(h, w, 4) int64 of ETC1s blocks: one 5-bit colour and one modifier table a block."""
    b = blocks.view(h // 4, w // 4, 8).to(torch.int64)
    c5 = b[..., :3] >> 3
    base = c5 << 3 | c5 >> 2
    small = torch.tensor([2, 5, 9, 13, 18, 24, 33, 47], device=b.device)[b[..., 3] >> 5]
    large = torch.tensor([8, 17, 29, 42, 60, 80, 106, 183], device=b.device)[b[..., 3] >> 5]
    mod = torch.stack([small, large, -small, -large], -1)
    msb, lsb = b[..., 4] << 8 | b[..., 5], b[..., 6] << 8 | b[..., 7]
    idx = torch.stack([(msb >> j & 1) << 1 | lsb >> j & 1 for j in range(16)], -1)  # pixel j = 4x + y
    px = (base[..., None, :] + torch.gather(mod, -1, idx)[..., None]).clamp(0, 255)
    px = torch.cat([px, torch.full(px.shape[:-1] + (1,), 255, dtype=torch.int64, device=b.device)], -1)
    return px.view(h // 4, w // 4, 4, 4, 4).permute(0, 3, 1, 2, 4).reshape(h, w, 4)


def exact(case, seed):
    """The quality record from its definition; every other case returns bytes and whole numbers only."""
    if case["kind"] != "quality":
        return None
    w, h = case["width"], case["height"]
    s = prepare(case, seed)
    torch.cuda.synchronize()
    px = (_decode_bc1 if case["codec"] == BC1 else _decode_etc1s)(s["blocks"], h, w)
    d = s["src"].to(torch.int64) - px
    n = w * h
    total = [int(v) for v in d.square().sum((0, 1)).cpu()]
    # a pixel read as a little-endian number: "r" is byte 2, "b" byte 0
    luma = int((21 * d[..., 2] + 72 * d[..., 1] + 7 * d[..., 0]).square().sum())

    def psnr(mse, peak):
        return sys.float_info.max if mse < 1e-7 else 10.0 * math.log10(peak * peak / mse)

    out = {"mse_b": total[0] / n, "mse_g": total[1] / n, "mse_r": total[2] / n, "mse_a": total[3] / n,
           "mse_rgb": sum(total[:3]) / n, "mse_y": luma / 10000.0 / n}
    out["mse_max"] = max(out["mse_" + c] for c in "rgba")
    for c in "rgbay":
        out["psnr_" + c] = psnr(out["mse_" + c], 255.0)
    out["psnr_min"] = min(out["psnr_" + c] for c in "rgba")
    out["psnr_rgb"] = psnr(out["mse_rgb"], 768.0)
    out["unsupported_blocks"] = 0
    return out
