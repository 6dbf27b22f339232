"""The forms of the SIMPLE pieces over components (fv_gpu.cu: each) on both
sides of the sizes where they change, bit for bit the host restatement; and
what the forms are for, as ratios of device times: a field of four components
costs less than as many scalars, and on a small mesh a vector field hardly
more than one."""
import numpy as np
import pytest

from programs_b200 import mesh as M
from programs_b200.mesh import Mesh

pytestmark = pytest.mark.gpu


def _d(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x, np.float64)).cuda()


def _same(a, b):
    return np.array_equal(a.cpu().numpy(), b)


@pytest.fixture(scope="module", params=[(25, 25, 25), (26, 25, 25), (40, 40, 40), (41, 41, 41)])
def case(request, built):
    from programs_b200.fv import GpuFv
    m = Mesh.hex(*request.param, jitter=0.2, seed=5, permute=True)
    m.renumber(Mesh.RCM)
    fv = GpuFv(m)
    yield m, fv
    fv.close()


@pytest.mark.parametrize("ncomp", [1, 2, 3, 4])
def test_sweeps_and_explicit_terms_are_the_host_s(case, ncomp):
    m, fv = case
    phi = M.uniform(3, ncomp * m.n_cell).reshape(-1, ncomp)
    phi = phi[:, 0].copy() if ncomp == 1 else phi
    wall = M.uniform(4, ncomp * m.n_face).reshape(-1, ncomp)
    flux = 0.01 * M.uniform(5, m.n_face)
    assert _same(fv.gradient(_d(phi)), M.gradient(m, phi))
    for n_iter, neu in ((1, 0), (2, 0), (3, 2)):
        g = M.gradient_sweeps(m, phi, n_iter, neu, wall if neu == 0 else None)
        assert _same(fv.gradient_sweeps(_d(phi), n_iter, neu, _d(wall) if neu == 0 else None), g)
    rhs = _d(np.zeros_like(phi))
    fv.momentum_deferred(_d(phi), _d(g), _d(flux), 2e-3, rhs, c_bl=0.9, scheme=2)
    assert _same(rhs, M.momentum_deferred(m, phi, g, flux, 2e-3, 0.9, 2))


@pytest.mark.parametrize("dims", [(84, 85, 84), (86, 85, 84)])
def test_gradient_of_a_vector_on_a_large_mesh(built, dims):
    from programs_b200.fv import GpuFv
    m = Mesh.hex(*dims, jitter=0.2, seed=5)
    fv = GpuFv(m)
    phi = M.uniform(3, 3 * m.n_cell).reshape(-1, 3)
    assert _same(fv.gradient(_d(phi)), M.gradient(m, phi))
    fv.close()


def _device_us(stream, f):
    """Median device time of one of 20 calls in a graph."""
    import torch
    f()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        for _ in range(20):
            f()
    t = []
    with torch.cuda.stream(stream):
        for k in range(14):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            g.replay()
            b.record()
            b.synchronize()
            t.append(a.elapsed_time(b) * 50.0)
    return float(np.median(t[3:]))


def test_components_share_what_they_read(built):
    """80^3, four components against one: 2.0 (3.75 with the components in
    blocks of their own); 9^3, two sweeps of a vector against a scalar: 1.0
    (1.43 with the components one after the other in a thread)."""
    import torch
    from programs_b200.fv import GpuFv
    for n, nc, most in ((80, 4, 2.8), (9, 3, 1.2)):
        m = Mesh.hex(n, jitter=0.15, seed=0, permute=True)
        m.renumber(Mesh.RCM)
        fv = GpuFv(m)
        st = torch.cuda.Stream()
        fv._lib.fv_gpu_set_stream(fv._h, st.cuda_stream)
        x = [_d(M.uniform(k, k * m.n_cell)) for k in (1, nc)]
        o = [torch.empty(3 * k * m.n_cell, dtype=torch.float64, device="cuda") for k in (1, nc)]
        t = []
        for k, a, b in zip((1, nc), x, o):
            if n == 80:
                t.append(_device_us(st, lambda: fv._lib.fv_gpu_gradient(
                    fv._h, k, a.data_ptr(), b.data_ptr())))
            else:
                t.append(_device_us(st, lambda: fv._lib.fv_gpu_gradient_sweeps(
                    fv._h, k, a.data_ptr(), None, 2, 2, b.data_ptr())))
        torch.cuda.synchronize()
        fv.close()
        assert t[1] < most * t[0], t
