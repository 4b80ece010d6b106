"""The synchronous quality calls keep accumulators per CUDA context: what a
context held is not used again once cudaDeviceReset has ended it."""
import ctypes
import glob
import os
import subprocess
import sys

import pytest

from goofy_gb300 import build as lib_build
from tests.host_emu import build as emu_build


@pytest.fixture(scope="module")
def slots(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("slots") / "libslots.so")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", lib_build.CSRC, "-o", so,
                           os.path.join(emu_build.HERE, "context_slots_host.cpp")])
    return ctypes.CDLL(so)


def test_a_new_context_finds_nothing_of_an_old_one(slots):
    swap = lambda i, v: slots.swap_value(ctypes.c_ulonglong(i), v)
    assert [swap(i, 10 * i) for i in (1, 2, 1, 2)] == [0, 0, 10, 20]  # two contexts in turn keep their own
    assert [swap(i, 10 * i) for i in (3, 4, 1, 3)] == [0, 0, 10, 30]
    assert swap(5, 50) == 0 and swap(2, 0) == 20 and swap(4, 0) == 40  # a fifth takes the oldest's slot
    assert swap(1, 11) == 0  # and the oldest starts anew, in that of 2
    assert swap(2, 22) == 0 and swap(5, 0) == 50


# Noise against blocks of zeros, measured before and after cudaDeviceReset (which ends only this
# process's context); the buffers after it are new ones.
CHILD = """
import ctypes, glob
import numpy as np
import goofy_gb300 as g
rt = ctypes.CDLL(%r)
def device(a):
    p = ctypes.c_void_p()
    assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(a.size)) == 0
    assert rt.cudaMemcpy(p, a.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(a.size), 1) == 0
    return p.value
for turn in range(3):
    assert rt.cudaFree(None) == 0
    for w, codec in ((64, 0), (64, 1), (1024, 0), (1024, 1)):  # the register-loading kernel and the ring
        rng = np.random.default_rng(w)
        img = rng.integers(0, 256, (w, 4 * w), np.uint8)
        blocks = np.zeros(w * w // 2, np.uint8)  # BC1: black; ETC1: individual mode, {2, 8, -2, -8} of black: 2
        rc, psnr, sums = g.psnr_rgb(codec, device(blocks), device(img), w, w, 4 * w)
        dec = np.array([2, 2, 2, 255] if codec else [0, 0, 0, 255])
        want = ((img.reshape(-1, 4).astype(np.int64) - dec) ** 2).sum(0).tolist()
        assert rc == g.OK and sums.tolist() == want + [0], (turn, w, codec, rc, sums, want, g.last_error())
    assert rt.cudaDeviceReset() == 0
print("same sums in three contexts")
"""


@pytest.mark.gpu
def test_quality_calls_after_a_device_reset(built):
    found = glob.glob(os.path.join(lib_build._cuda_home(), "lib64", "libcudart.so.*"))
    if not found:
        pytest.skip("no libcudart")
    env = dict(os.environ, GOOFY_TILE_CACHE="")
    r = subprocess.run([sys.executable, "-c", CHILD % found[0]], cwd=emu_build.ROOT, env=env, capture_output=True,
                       text=True, timeout=120)
    assert r.returncode == 0 and "same sums" in r.stdout, r.stdout + r.stderr
