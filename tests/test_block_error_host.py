"""The quality kernels' per-block error sums (goofy_gb300/csrc/block_error.cuh),
compiled for the CPU with emulated intrinsics, against the oracle's decoder
and integer sums: every block mode, extreme pixels, random alpha."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import oracle
from tests.host_emu import build as emu_build

SO = os.path.join(emu_build.HERE, "_build", "libblock_error_host.so")
CSRC = os.path.join(emu_build.ROOT, "goofy_gb300", "csrc")


@pytest.fixture(scope="module")
def emu(built):
    os.makedirs(os.path.dirname(SO), exist_ok=True)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-DGOOFY_HOST_EMULATION", "-I",
                           emu_build.HERE, "-I", CSRC, "-o", SO, os.path.join(emu_build.HERE, "block_error_host.cpp")])
    lib = ctypes.CDLL(SO)
    lib.host_emu_errors.restype = None
    lib.host_emu_errors.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint, ctypes.c_uint,
                                    ctypes.c_uint, ctypes.c_uint, ctypes.c_void_p]
    return lib


def _check(emu, codec, blocks, img, w, h, every=2048):
    got = np.zeros(6, np.uint64)
    blocks = np.ascontiguousarray(blocks)
    emu.host_emu_errors(codec, blocks.ctypes.data, img.ctypes.data, w, h, img.strides[0], every, got.ctypes.data)
    px, bad = oracle.decode(codec, blocks, w, h)
    d = img.reshape(h, w, 4).astype(np.int64) - px.reshape(h, w, 4).astype(np.int64)
    want = [int((d[..., c] ** 2).sum()) for c in range(4)]
    luma = int(((21 * d[..., 2] + 72 * d[..., 1] + 7 * d[..., 0]) ** 2).sum())
    assert [int(v) for v in got] == want + [bad, luma]


@pytest.mark.parametrize("codec", [0, 1])
@pytest.mark.parametrize("pixels", ["random", "extreme", "zero", "full"])
def test_random_blocks_of_every_mode(emu, codec, pixels):
    rng = np.random.default_rng(31 + codec)
    w, h = 512, 256
    blocks = rng.integers(0, 256, (w // 4) * (h // 4) * 8, dtype=np.uint8)
    img = {"random": rng.integers(0, 256, (h, 4 * w)), "extreme": 255 * rng.integers(0, 2, (h, 4 * w)),
           "zero": np.zeros((h, 4 * w)), "full": np.full((h, 4 * w), 255)}[pixels].astype(np.uint8)
    _check(emu, codec, blocks, img, w, h)


@pytest.mark.parametrize("codec", [0, 1])
def test_encoded_blocks(emu, codec):
    rng = np.random.default_rng(5)
    w, h = 256, 256
    for amp in (255, 40, 1):
        img = np.clip(rng.integers(0, 256, (h // 4, w // 4, 1, 1, 4)) + rng.integers(-amp, amp + 1, (h // 4, w // 4, 4, 4, 4)),
                      0, 255).astype(np.uint8)
        img = np.ascontiguousarray(img.transpose(0, 2, 1, 3, 4).reshape(h, 4 * w))
        _check(emu, codec, oracle.encode(codec, img, w, h), img, w, h)


@pytest.mark.parametrize("codec", [0, 1])
def test_sums_at_their_bound(emu, codec):
    """2048 blocks of the largest differences before a flush: black blocks under white pixels and the reverse."""
    w, h = 256, 512
    n = (w // 4) * (h // 4)
    black = np.zeros((n, 8), np.uint8)
    if codec == 1:
        black[:, 3] = 2  # differential, zero deltas
    white = np.zeros((n, 8), np.uint8)
    white[:, :4] = 0xFF if codec == 0 else (0xF8, 0xF8, 0xF8, 0xFE)
    for blocks in (black, white):
        for value in (0, 255):
            _check(emu, codec, blocks, np.full((h, 4 * w), value, np.uint8), w, h)
