"""What is set once per device (function attributes, occupancies) is made by the first call on
each device of the process, and once (qz_test_per_device; no GPU needed)."""
import ctypes as C

import pytest

from quantizer_b200 import core


@pytest.mark.parametrize("devices,made", [([], 0), ([0], 1), ([0, 0, 0], 1), ([0, 1], 2),
                                          ([1, 0, 7, 0, 1, 7, 2], 4)])
def test_each_device_is_set_up_once(devices, made):
    assert core.load().qz_test_per_device((C.c_int * len(devices))(*devices), len(devices)) == made
