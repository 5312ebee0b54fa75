"""The allocation-free direct sum allocates nothing at any size it routes differently (GPU).

In a process of its own, so that no earlier call has loaded a kernel (kernels are
loaded at their first launch): after the count-0 call, calls of each size (the
target counts per CTA of the small-system kernel, one and two targets per thread of the general one, with and
without softening, and accelerations in the place of an input) leave the free device memory as it is.
"""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

from conftest import PKG_DIR

pytestmark = pytest.mark.gpu

CODE = """
import ctypes as C, sys
sys.path.insert(0, sys.argv[1])
import torch
import nbgb as nb
torch.zeros(1, device="cuda")
fn = nb.lib().nbgb_compute_forces_direct_noalloc
fn.restype, fn.argtypes = C.c_int, [C.c_void_p, C.c_float, C.c_float, C.c_void_p]
sizes = (1, 1000, 2000, 4000, 5000, 9000, 20000, 65536)
data = []
for n in sizes:
    s = nb.ics.plummer(n, seed=n)
    data.append(nb.ScopedParticleData(n, {"pos_x": s["x"], "pos_y": s["y"], "pos_z": s["z"],
                                          "mass": s["m"]}))
empty = nb.ParticleData()
assert fn(C.addressof(empty.struct), 1.0, 0.01, None) == 0
torch.cuda.synchronize()
free0 = torch.cuda.mem_get_info()[0]
for eps in (0.01, 0.0):
    for n, p in zip(sizes, data):
        assert fn(C.addressof(p.device.struct), 1.0, eps, None) == 0
        free1 = torch.cuda.mem_get_info()[0]
        assert free1 == free0, (n, eps, free0 - free1)
for n, p in zip(sizes, data):  # accelerations over the positions
    p.device.struct.acc_x = p.device.struct.pos_x
    assert fn(C.addressof(p.device.struct), 1.0, 0.01, None) == 0
    free1 = torch.cuda.mem_get_info()[0]
    assert free1 == free0, (n, "in place", free0 - free1)
import os
os._exit(0)  # (pointers were exchanged: the arrays are not freed one by one)
"""


def test_no_size_allocates_after_the_warm_up(nb):
    env = dict(os.environ, CUDA_MODULE_LOADING="LAZY")
    r = subprocess.run([sys.executable, "-c", CODE, PKG_DIR], capture_output=True, text=True,
                       timeout=300, env=env)
    assert r.returncode == 0, r.stdout + r.stderr
