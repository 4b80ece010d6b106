"""A quality measurement whose kernel left blocks out (a bounded wait gave up)
is no result: the kernel's end reports it with the totals and the synchronous
calls return an error.  No wait runs out here: the report is made up."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from goofy_gb300 import build as lib_build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("handover") / "libhandover.so")
    subprocess.check_call([lib_build._nvcc(), "-O1", "-std=c++17", *lib_build.ARCH, "-shared", "-Xcompiler", "-fPIC",
                           "-I", lib_build.CSRC, "-I", lib_build.INCLUDE, "-o", so,
                           os.path.join(HERE, "error_handover.cu")])
    return ctypes.CDLL(so)


def _u64(*v):
    return np.array(v, np.uint64)


@pytest.mark.parametrize("count", [0, 1, (1 << 31) - 1])
@pytest.mark.parametrize("warps", [0, 1, 16 * 2048])
def test_totals_are_complete_unless_a_warp_gave_up(lib, count, warps):
    totals = _u64(7, 7, 7, 7, count + (warps << 40), 7)
    assert lib.complete_totals(ctypes.c_void_p(totals.ctypes.data)) == (warps == 0)


@pytest.mark.gpu
@pytest.mark.parametrize("ctas,gave_up", [(1, 0), (1, 1), (3, 0), (3, 0b0001_0000_1000), (8, 0xFFFFFFFF)])
@pytest.mark.parametrize("host", [1, 0])
def test_the_kernel_reports_warps_that_gave_up(cuda, lib, ctas, gave_up, host):
    totals = np.zeros(6, np.uint64)
    rc = lib.handover(ctas, ctypes.c_uint(gave_up), host, ctypes.c_void_p(totals.ctypes.data))
    n = 128 * ctas
    reported = bin(gave_up).count("1") if host else 0  # a caller's accumulator holds the count alone
    luma = n * (441 * 3 + 5184 * 2 + 49 * 1)
    assert totals.tolist() == [n, 2 * n, 3 * n, 4 * n, n + (reported << 40), luma]
    assert rc == (reported == 0)
