"""dump_bytes without a GPU: no records need none."""
import ctypes

import numpy as np

import ktcountermemorygreedy_b200 as kc


def test_dump_leaves_the_interpreters_prototypes_alone():
    """ctypes.pythonapi is shared by the whole process."""
    f = ctypes.pythonapi.PyBytes_FromStringAndSize
    before = f.argtypes, f.restype
    assert kc.dump_bytes(np.zeros(0, np.uint64), np.zeros(0, np.uint32), 31) == b""
    assert (f.argtypes, f.restype) == before
