"""Host buffers that only offer numpy's `ctypes` attribute."""
import numpy as np

import goofy_gb300 as g


class Wrapped:
    """An array's owner that passes on its `ctypes` attribute and nothing else."""

    def __init__(self, a):
        self.a = a

    @property
    def ctypes(self):
        return self.a.ctypes


def test_an_object_with_only_the_ctypes_attribute():
    for a in (np.zeros(64, np.uint8), np.zeros((4, 32), np.uint8)[:, 8:], np.frombuffer(bytes(8), np.uint8)):
        assert g._addr(Wrapped(a)) == a.ctypes.data
