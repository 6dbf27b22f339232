"""The SIMPLE pieces on the GPU over component counts and mesh shapes where
their forms change: three components in one thread, any other count one per
thread; slices of 32 cells that end ragged or hold boundary cells only.  Bit
for bit the host restatement, as tests/test_gpu_fv.py."""
import numpy as np
import pytest

from programs_b200 import mesh as M
from programs_b200.mesh import Mesh

pytestmark = pytest.mark.gpu


def _d(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x, np.float64)).cuda()


@pytest.mark.parametrize("dims", [(1, 1, 1), (1, 3, 2), (4, 8, 1), (5, 7, 3), (11, 9, 13)])
@pytest.mark.parametrize("ncomp", [1, 2, 3, 5])
def test_gradients_and_explicit_terms(built, dims, ncomp):
    from programs_b200.fv import GpuFv
    m = Mesh.hex(*dims, jitter=0.2, seed=5, permute=True)
    m.renumber(Mesh.RCM)
    fv = GpuFv(m)
    phi = M.uniform(3, ncomp * m.n_cell).reshape(-1, ncomp)
    phi = phi[:, 0].copy() if ncomp == 1 else phi
    wall = M.uniform(4, ncomp * m.n_face).reshape(-1, ncomp)
    flux = 0.01 * M.uniform(5, m.n_face)
    same = lambda a, b: np.array_equal(a.cpu().numpy(), b)
    assert same(fv.gradient(_d(phi)), M.gradient(m, phi))
    for n_iter, neu in ((1, 0), (2, 0), (2, 1), (3, 2)):
        g = M.gradient_sweeps(m, phi, n_iter, neu, wall if neu == 0 else None)
        assert same(fv.gradient_sweeps(_d(phi), n_iter, neu, _d(wall) if neu == 0 else None), g)
    for scheme in range(4):
        rhs = _d(np.zeros_like(phi))
        fv.momentum_deferred(_d(phi), _d(g), _d(flux), 2e-3, rhs, c_bl=0.9, scheme=scheme)
        assert same(rhs, M.momentum_deferred(m, phi, g, flux, 2e-3, 0.9, scheme))
    fv.close()
