"""A flow that meets a full device: refused for want of memory for its kernels
or its step graph, it leaves the links it was given, and says so once.  In a
process of its own, whose kernels are not loaded yet, beside a filler that holds
what memory is left."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import sys
sys.path.insert(0, sys.argv[1])
kind, precision = sys.argv[2], sys.argv[3]
import ctypes
import numpy as np
import torch
from latticeyangmills_b200 import Ensemble, YmflowError

SIZES = {"runs": [(8, 8, 8, 6 + k) for k in range(6)], "list": [(8, 8, 8, 8)] * 3}
sizes = SIZES[kind]


def make():
    f = Ensemble(sizes, precision)
    for c in range(len(sizes)):
        f.init_links(c, "expiah", 0.35, 1 + c)
    if kind == "runs":
        f.set_tuning(3)
    return f


def links(f):
    return [f.download(c) for c in range(len(sizes))]


f = make()
f.flow(0.01, 0, 0)
before = links(f)
torch.zeros(1, device="cuda")
runtime = ctypes.CDLL("libcudart.so.12")  # torch's
filler, size = [], 1 << 35
while size >= 1 << 16 and len(filler) < 4000:  # room for rows, none for a kernel
    p = ctypes.c_void_p()
    if runtime.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(size)) == 0:
        filler.append(p)
    else:
        runtime.cudaGetLastError()
        size >>= 1
try:
    f.flow(0.01, 6, 0)
    refused = False
except YmflowError as e:
    print("refused:", e)
    refused = True
for p in filler:
    runtime.cudaFree(p)
after = links(f)  # an error left over from the refusal would be reported here
if refused:
    want = before
else:
    g = make()
    g.flow(0.01, 6, 0)
    want = links(g)
for a, b in zip(after, want):
    assert np.array_equal(a, b), "a refused flow changed the links" if refused else "other links beside the filler"
print("ok")
"""


@pytest.mark.parametrize("kind", ["runs", "list"])
@pytest.mark.parametrize("precision", ["fp64", "fp32_12"])
def test_a_full_device_leaves_the_links(kind, precision):
    res = subprocess.run([sys.executable, "-c", SCRIPT, str(ROOT), kind, precision], capture_output=True, text=True,
                         timeout=300)
    print(res.stdout)
    assert res.returncode == 0, res.stdout + res.stderr[-2000:]
