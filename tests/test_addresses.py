"""The addresses the Python layer passes for host buffers: arrays of every
layout give numpy's own data pointer."""
import ctypes

import numpy as np
import pytest

import goofy_gb300 as g


@pytest.mark.parametrize("make", [
    lambda: np.zeros(64, np.uint8),
    lambda: np.zeros((4, 16), np.uint8),
    lambda: np.zeros((4, 32), np.uint8)[:, :16],        # rows with a gap
    lambda: np.zeros((4, 16), np.uint8)[1:, 3:],        # starts inside
    lambda: np.zeros((4, 16), np.uint8).T,
    lambda: np.frombuffer(bytes(64), np.uint8),         # read-only
    lambda: np.zeros(0, np.uint8),
    lambda: np.zeros((2, 3), np.float64),
    lambda: np.zeros(3, "datetime64[s]"),
    lambda: np.zeros((4, 16), np.uint8)[::-1],
])
def test_numpy_arrays(make):
    a = make()
    assert g._addr(a) == a.ctypes.data


def test_other_buffers():
    raw = bytearray(16)
    assert g._addr(raw) == ctypes.addressof((ctypes.c_char * 16).from_buffer(raw))
    c = (ctypes.c_uint8 * 8)()
    assert g._addr(c) == ctypes.addressof(c)
    assert g._addr(None) is None and g._addr(12345) == 12345


def test_an_array_can_be_resized_after_its_address_was_taken():
    a = np.zeros(64, np.uint8)
    g._addr(a)
    a.resize(128, refcheck=False)  # no exported buffer is left behind
    raw = bytearray(8)
    g._addr(raw)
    raw.extend(b"12345678")
