"""Blocks read with their columns x in the places x ^ q (word-aligned rows):
the same blocks, bit for bit, as the oracle's from the columns in order."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import oracle
from tests.host_emu import build as emu_build

SO = os.path.join(emu_build.HERE, "_build", "libblock_columns_host.so")
CSRC = os.path.join(emu_build.ROOT, "goofy_gb300", "csrc")


@pytest.fixture(scope="module")
def emu(built):
    os.makedirs(os.path.dirname(SO), exist_ok=True)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-DGOOFY_HOST_EMULATION", "-I",
                           emu_build.HERE, "-I", CSRC, "-o", SO, os.path.join(emu_build.HERE, "block_columns_host.cpp")])
    lib = ctypes.CDLL(SO)
    lib.host_emu_encode_columns.restype = None
    lib.host_emu_encode_columns.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint, ctypes.c_uint]
    return lib


@pytest.mark.parametrize("q", range(4))
@pytest.mark.parametrize("amp", [255, 40, 3])
def test_columns_in_any_place(emu, q, amp):
    rng = np.random.default_rng(amp)
    n = 1 << 14
    px = np.clip(rng.integers(0, 256, (n, 1, 4)) + rng.integers(-amp, amp + 1, (n, 16, 4)), 0, 255).astype(np.uint8)
    img = np.ascontiguousarray(px.reshape(n, 4, 16).transpose(1, 0, 2).reshape(4, 16 * n))  # one row of blocks
    want = [oracle.encode(codec, img, 4 * n, 4).reshape(n, 8) for codec in (0, 1)]
    for codec in (0, 1):
        got = np.zeros((n, 8), np.uint8)
        emu.host_emu_encode_columns(codec, got.ctypes.data, px.ctypes.data, n, q)
        np.testing.assert_array_equal(got, want[codec])
    got = np.zeros((n, 16), np.uint8)
    emu.host_emu_encode_columns(2, got.ctypes.data, px.ctypes.data, n, q)
    np.testing.assert_array_equal(got, np.hstack(want))
