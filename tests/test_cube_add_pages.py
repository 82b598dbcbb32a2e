"""Page faults of the native pass into a fresh host array, as np.zeros hands
one to the first insertion: one for a page (its first write), not a read fault
and a write fault, however many threads share the work (CPU only)."""

import mmap
import os
import resource

import numpy as np
import pytest

from martini_gb300.martini import add_to_array

LINUX = tuple(int(p) for p in os.uname().release.split("-")[0].split(".")[:2])
pytestmark = pytest.mark.skipif(not hasattr(mmap, "MADV_NOHUGEPAGE") or LINUX < (5, 14),
                                reason="needs MADV_NOHUGEPAGE and MADV_POPULATE_WRITE")


@pytest.mark.parametrize("divide_all", [True, False])
@pytest.mark.parametrize("shape", [(128, 128, 128), (301, 37, 130), (1, 900, 700), (700, 900, 1)])
def test_one_fault_a_page(shape, divide_all):
    n = int(np.prod(shape))
    buf = mmap.mmap(-1, n * 8, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS)
    buf.madvise(mmap.MADV_NOHUGEPAGE)
    arr = np.frombuffer(buf, dtype=np.float64).reshape(shape)
    add = np.full(shape, 0.5, np.float32)
    add_to_array(np.zeros((2, 2, 2)), np.zeros((2, 2, 2), np.float32), (0, 0), 1.0, True)
    before = resource.getrusage(resource.RUSAGE_SELF).ru_minflt
    add_to_array(arr, add, (0, 0), 2.0, divide_all)
    faults = resource.getrusage(resource.RUSAGE_SELF).ru_minflt - before
    pages = n * 8 // mmap.PAGESIZE
    sums = shape[0] * shape[2] * 8 // mmap.PAGESIZE  # the rows' sums
    # eight threads' stacks and heaps beside the two
    assert faults <= pages + sums + 300, (faults, pages)
    assert np.all(arr == 0.25)
