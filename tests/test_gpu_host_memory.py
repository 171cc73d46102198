"""What the calls on a caller's arrays leave behind in its memory."""
import ctypes
import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _vm_flags(addr):
    """The kernel's flags of the mapping that holds addr."""
    inside = False
    for line in open("/proc/self/smaps"):
        head = line.split()[0]
        if "-" in head and not head.endswith(":"):
            lo, hi = (int(x, 16) for x in head.split("-"))
            inside = lo <= addr < hi
        elif inside and head == "VmFlags:":
            return line.split()[1:]
    return []


def test_sorting_in_place_leaves_the_mapping_as_it_was():
    """Arrays in a mapping of the caller's, sorted in place: its advice for huge
    pages is the caller's to give."""
    import ktcountermemorygreedy_b200 as kc
    n = 2_000_000
    m = mmap.mmap(-1, 32 << 20)
    keys = np.frombuffer(m, np.uint64, n)
    counts = np.frombuffer(m, np.uint32, n, offset=8 * n)
    rng = np.random.default_rng(1)
    keys[:] = rng.permutation(n)
    counts[:] = keys % 1000
    addr = keys.ctypes.data + (16 << 20)
    before = _vm_flags(keys.ctypes.data)
    assert before and "hg" not in before
    rc = kc.lib().kc_sort_records(ctypes.c_void_p(keys.ctypes.data), ctypes.c_void_p(counts.ctypes.data), n, 40)
    assert rc == 0 and np.array_equal(keys, np.arange(n)) and np.array_equal(counts, np.arange(n) % 1000)
    for a in (keys.ctypes.data, keys.ctypes.data + (4 << 20), addr):
        assert "hg" not in _vm_flags(a)


@pytest.mark.parametrize("n", [900_000, 1_100_000])
def test_dump_on_both_sides_of_the_advice(n):
    """Texts below and above 32 MiB."""
    import ktcountermemorygreedy_b200 as kc
    rng = np.random.default_rng(n)
    keys, counts = np.sort(rng.integers(0, 1 << 60, n, dtype=np.uint64)) << np.uint64(2), np.full(n, 77, np.uint32)
    text = kc.dump_bytes(keys, counts, 31)
    assert len(text) == n * 35 and text.count(b"\t77\n") == n
    lines = text.split(b"\n")
    for i in range(0, n, 9973):
        s = "".join("ACGT"[(int(keys[i]) >> (2 + 2 * b)) & 3] for b in range(31))
        assert lines[i] == f"{s}\t77".encode()
