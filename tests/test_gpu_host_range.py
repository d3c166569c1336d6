"""GPU: qz_step_host lets a kernel read host arrays only where each is page-locked as a whole
(qz_test_host_range, the question it asks): registered in part, past the end of a
registration, pageable, and whole allocations of either kind.  Nothing is read here."""
import mmap

import numpy as np
import torch
import pytest

from quantizer_b200 import core

pytestmark = pytest.mark.gpu

PAGE = mmap.PAGESIZE


def test_a_range_is_page_locked_as_a_whole_or_not():
    lib = core.load()
    torch.cuda.init()
    mem = mmap.mmap(-1, 8 * PAGE)
    at = np.frombuffer(mem, dtype=np.uint8).ctypes.data
    assert lib.qz_test_host_range(at, 8) == 0
    rt = torch.cuda.cudart()
    assert int(rt.cudaHostRegister(at + 2 * PAGE, 3 * PAGE, 0)) == 0
    try:
        assert lib.qz_test_host_range(at, 8) == 0
        assert lib.qz_test_host_range(at + 2 * PAGE, 3 * PAGE) == 1
        assert lib.qz_test_host_range(at + 3 * PAGE + 8, 2 * PAGE - 8) == 1
        assert lib.qz_test_host_range(at + 2 * PAGE, 3 * PAGE + 1) == 0
        assert lib.qz_test_host_range(at + 4 * PAGE, 2 * PAGE) == 0
        assert lib.qz_test_host_range(at + 5 * PAGE, 8) == 0
    finally:
        assert int(rt.cudaHostUnregister(at + 2 * PAGE)) == 0


def test_whole_allocations():
    lib = core.load()
    torch.cuda.init()
    for n in (1, 1000, 32768):
        a = torch.empty(n, dtype=torch.float64, pin_memory=True)
        assert lib.qz_test_host_range(a.data_ptr(), 8 * n) == 1
