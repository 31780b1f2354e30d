"""A host program may reset the device between two uses of the library
(cudaDeviceReset ends the process's context on it).  What the kernels need of
the context, such as the cluster size and the shared memory they are allowed,
must be there again.  In a process of its own; the reset comes through the
CUDA runtime that torch has loaded."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes as C, sys
import torch
sys.path.insert(0, {root!r})
import numpy as np
from adcirc_b200 import model

def go(prec):
    g = model.GpuModel(model.channel_case(), prec)
    its, _ = g.run(1, 5)
    g.close()
    return list(map(int, its))

a = [go(0), go(18)]
rt = [line.split()[-1] for line in open("/proc/self/maps") if "libcudart" in line][0]
assert C.CDLL(rt).cudaDeviceReset() == 0
b = [go(0), go(18)]
assert a == b, (a, b)
print("same", a)
"""


def test_contexts_after_a_device_reset():
    import pathlib
    root = str(pathlib.Path(__file__).resolve().parents[1])
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=root)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr
