"""Device memory between handles: what a host that resets the device may expect."""
import os
import subprocess
import sys

import pytest

from gdon3d_b200 import capi, kuhn

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

RESET = r"""
import ctypes, glob, os, sys
sys.path.insert(0, %r)
import conftest
from gdon3d_b200 import capi, kuhn
import numpy as np
found = []
for p in sys.path:
    found += glob.glob(os.path.join(p, "nvidia", "cuda_runtime", "lib", "libcudart.so*"))
found += glob.glob("/usr/local/cuda/lib64/libcudart.so*")
rt = ctypes.CDLL(sorted(found)[0])
small = capi.mesh_build(*kuhn.kuhn_cube(3, 0.1, seed=1))
large = capi.mesh_build(*kuhn.kuhn_cube(40, 0.1, seed=1))  # blocks above the pool's (kinetic: 1.2 GB)
first = None
for k in range(3):
    out = []
    for mesh, scheme in ((small, capi.SCHEME_RK3), (small, capi.SCHEME_KINETIC), (large, capi.SCHEME_KINETIC)):
        s = capi.Solver(mesh, scheme, capi.plane_data(), 1e-3, rk3_variant=1, kin_sweep=1)
        out.append(s.solve(2)[0])
        s.close()
    assert first is None or all(np.array_equal(a, b) for a, b in zip(out, first)), k
    first = out
    assert rt.cudaDeviceReset() == 0
print("RESET OK")
"""


def test_attach_after_a_device_reset():
    r = subprocess.run([sys.executable, "-c", RESET % HERE], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "RESET OK" in r.stdout, r.stdout + r.stderr


def _free():
    import torch
    return torch.cuda.mem_get_info(0)[0]


def test_kept_memory_is_given_back():
    """After the last detach up to 1 GiB is kept; the release call returns it."""
    mesh = capi.mesh_build(*kuhn.kuhn_cube(32, 0.1, seed=1))

    def once():
        s = capi.Solver(mesh, dt=1e-4)  # 0.4 GiB, all in pool blocks
        s.solve(2)
        s.close()

    once()  # kernels are loaded with their first launch
    capi.release_memory()
    before = _free()
    once()
    kept = before - _free()
    assert 0 < kept <= 1 << 30
    capi.release_memory()
    assert _free() == before
    once()  # and the next attach takes it anew
