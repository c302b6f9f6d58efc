"""What a kernel keeps between launches is kept per device.

A kernel's shared-memory limit and the blocks a device holds belong to the
device: found once for a process, they left every device after the first with
the default limit, and the persistent step kernels did not launch there.
"""
import ctypes
import os
import re

import numpy as np
import pytest

from imexlb_b200 import api

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "imexlb_b200", "csrc")


# (64 and -1: outside the table, found each time)
@pytest.mark.parametrize("devices,found", [([0, 0, 0], 1), ([0, 1, 0, 1], 2), ([3, 0, 63, 3, 63], 3), ([64, 64, -1], 3)])
def test_each_device_has_its_own_number(devices, found):
    fn = api.load_library().imexlb_debug_per_device
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
    dev = np.array(devices, dtype=np.int32)
    got = np.zeros_like(dev)
    assert fn(dev.ctypes.data, len(devices), got.ctypes.data) == found
    assert got.tolist() == [100 + d for d in devices]


def test_no_launch_keeps_a_number_for_the_whole_process():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as fh:
                assert not re.findall(r"\bstatic int \w+ = ", fh.read()), name
