"""A cell with very many faces (a plenum that all the others open into): the
lists of its slice of 32 cells are as long as its own.  The entry point takes
such a mesh as far as memory goes, and where memory ends it says so instead of
throwing through the C call; on the GPU the results are those of the faces
added in ascending order."""
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# 70 million faces: 2.2e9 slots of 8 bytes.  Within 10 GB of address space the
# answer is SOLV_GPU_TOO_LARGE (9); SOLV_GPU_BAD_INPUT (4) would refuse the mesh.
CHILD = """
import ctypes, resource, sys
import numpy as np
sys.path.insert(0, %r)
resource.setrlimit(resource.RLIMIT_AS, (10 << 30, 10 << 30))
from programs_b200.solver import lib
n = 70_000_000
ip, inb = np.ones(n, np.int32), np.zeros(n, np.int32)
d = np.zeros(8)
h = ctypes.c_void_p()
f = lib().fv_gpu_create
f.argtypes = [ctypes.POINTER(ctypes.c_void_p)] + [ctypes.c_int] * 3 + [ctypes.c_void_p] * 9
print(f(ctypes.byref(h), 0, 2, n, ip.ctypes.data, inb.ctypes.data, *[d.ctypes.data] * 7))
"""


def test_a_mesh_beyond_memory_is_answered(built):
    r = subprocess.run([sys.executable, "-c", CHILD % ROOT], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.split()[-1:] == ["9"], (r.returncode, r.stdout, r.stderr)


class _Star:
    """Cell 1 owns a face to every other cell; geometry by seed."""

    def __init__(self, n):
        rng = np.random.default_rng(n)
        self.n_cell, self.n_face = n, n - 1
        self.ip, self.inb = np.ones(n - 1, np.int32), np.arange(2, n + 1, dtype=np.int32)
        self.nrm = rng.uniform(-1, 1, (n - 1, 3))
        self.s, self.l, self.w = rng.uniform(0.2, 1, (3, n - 1))
        self.xf, self.xc = rng.uniform(-1, 1, (n - 1, 3)), rng.uniform(-1, 1, (n, 3))
        self.vol = rng.uniform(0.5, 1, n)

    def faces(self):
        return self.ip, self.inb

    def face_geom(self):
        return self.s, self.nrm, self.xf, self.l, self.w

    def cell_geom(self):
        return self.xc, self.vol


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1000, 40001])
def test_hub_sums_run_in_face_order(built, n):
    import torch
    from programs_b200.fv import GpuFv
    m = _Star(n)
    fv = GpuFv(m)
    phi = np.random.default_rng(1).uniform(-1, 1, (n, 2))
    got = fv.gradient(torch.from_numpy(phi).cuda()).cpu().numpy()
    flux = np.random.default_rng(2).uniform(-1, 1, n - 1)
    b, _ = fv.mass_imbalance(torch.from_numpy(flux).cuda(), pin=0)
    fv.close()
    pf = m.w[:, None] * phi[1:] + (1.0 - m.w)[:, None] * phi[0]
    t = (pf * m.s[:, None])[:, :, None] * m.nrm[:, None, :]
    assert np.array_equal(got[0], np.cumsum(t, axis=0)[-1] / m.vol[0])  # one after the other
    assert np.array_equal(got[1:], (0.0 - t) / m.vol[1:, None, None])
    assert b[0].item() == np.cumsum(-flux)[-1]
    assert np.array_equal(b[1:].cpu().numpy(), flux)
