"""A launch that the CUDA runtime refuses (solv_gpu_selftest_fail_launch gives
the answer on the host; nothing reaches the GPU) ends the call with
DEVICE_ERROR wherever in an iteration it stood, and leaves nothing behind: no
graph without that kernel, no error for the next call to report, no half-used
sweep buffers.  The solve that follows is the one a context never disturbed
makes."""
import numpy as np
import pytest

from programs_b200 import learn
from programs_b200.mesh import Mesh, uniform
from programs_b200.solver import (DEVICE_ERROR, OK, OPT_BLOCK, OPT_GNN_LOSS, OPT_GRAPH_ITERS,
                                  OPT_GRAPH_LOOP, OPT_PRECISION, SolverError)

pytestmark = pytest.mark.gpu
OUT_OF_RESOURCES = 701  # cudaErrorLaunchOutOfResources


@pytest.fixture(scope="module")
def system(gpu):
    m = Mesh.hex(30, jitter=0.15, seed=2, permute=True)
    m.renumber(Mesh.RCM)
    gpu.gnn_set_params(learn.load_params())
    return m.pressure(pin=1), m.momentum()[0]


def _solver(gpu, system, kind, precision):
    A = system[kind == "bicg"]
    gpu.matrix_set(A)
    b = uniform(3, A.n_cell)
    b -= b.mean()
    b = b.reshape(-1, 1)

    def solve():
        gpu.set_option(OPT_BLOCK, 256)  # the graphs are captured again
        gpu.set_option(OPT_PRECISION, precision)
        phi, res = np.zeros(b.shape), np.asfortranarray(b.copy())
        if kind == "fcg":
            st = gpu.solv_fcg(1e-10, 2000, phi, res, np.zeros(1))
        else:
            st = getattr(gpu, "solv_" + kind)(1 if kind == "cg" else 2, 1e-10, 2000, phi, res,
                                              np.zeros(1))
        return phi, st
    return solve


@pytest.mark.parametrize("kind,precision,loop,iters", [
    ("fcg", 1, 2, 16), ("fcg", 1, 0, 2), ("cg", 0, 0, 2), ("cg", 1, 0, 0), ("bicg", 1, 1, 2)])
def test_refused_launches_in_a_solve(gpu, system, kind, precision, loop, iters):
    solve = _solver(gpu, system, kind, precision)
    gpu.set_option(OPT_GRAPH_LOOP, loop)
    gpu.set_option(OPT_GRAPH_ITERS, iters)
    try:
        phi0, st0 = solve()
        assert st0["status"] == OK
        refused = 0
        for nth in range(1, 30):
            gpu.selftest_fail_launch(nth, OUT_OF_RESOURCES)
            try:
                solve()
            except SolverError as e:
                assert e.code == DEVICE_ERROR
                refused += 1
            else:
                assert iters  # all the launches of a graph are passed
                break
            finally:
                gpu.selftest_fail_launch(0)
            phi, st = solve()
            assert st["status"] == OK and st["fallbacks"] == st0["fallbacks"]
            assert abs(st["iters"][0] - st0["iters"][0]) <= 2
            assert np.linalg.norm(phi - phi0) <= 1e-8 * np.linalg.norm(phi0)
        assert refused >= 6
    finally:
        gpu.set_option(OPT_GRAPH_LOOP, 2)
        gpu.set_option(OPT_GRAPH_ITERS, 16)
        gpu.set_option(OPT_PRECISION, 0)


def test_refused_launches_in_a_training_step(gpu, system):
    import torch
    A = system[0]
    gpu.matrix_set(A)
    gpu.set_option(OPT_GNN_LOSS, 2)
    r = torch.from_numpy(uniform(5, A.n_cell)).cuda()
    try:
        loss0 = gpu.gnn_grad_dev(r.data_ptr(), r.data_ptr(), 1)
        refused = 0
        for nth in range(1, 40):
            gpu.selftest_fail_launch(nth, OUT_OF_RESOURCES)
            try:
                gpu.gnn_grad_dev(r.data_ptr(), r.data_ptr(), 1)
            except SolverError as e:
                assert e.code == DEVICE_ERROR
                refused += 1
            else:
                break
            finally:
                gpu.selftest_fail_launch(0)
            assert abs(gpu.gnn_grad_dev(r.data_ptr(), r.data_ptr(), 1) - loss0) <= 1e-5 * abs(loss0)
        assert refused >= 6
    finally:
        gpu.set_option(OPT_GNN_LOSS, 1)


@pytest.mark.parametrize("persistent", [0, 1])
def test_a_resident_launch_too_large_for_the_gpu(gpu, persistent):
    """Where the resident PCG's blocks cannot all run at once the solve takes
    the form it would have without it: step kernels, or a cluster."""
    from oracle.oracle import Oracle
    from programs_b200.mesh import poisson_rhs
    from programs_b200.solver import OPT_PERSISTENT
    too_large = 720  # cudaErrorCooperativeLaunchTooLarge
    m = Mesh.hex(24, jitter=0.15, seed=2, permute=True)
    m.renumber(Mesh.RCM)
    A = m.pressure(pin=1)
    b = poisson_rhs(A.n_cell, 4).reshape(-1, 1)
    ref = Oracle.from_matrix(A).solv_cg(0, 1e-10, 5000, np.zeros((A.n_cell, 1)), b)
    gpu.matrix_set(A)
    gpu.set_option(OPT_PERSISTENT, persistent)

    def solve():
        phi, res = np.zeros((A.n_cell, 1)), np.asfortranarray(b.copy())
        st = gpu.solv_cg(0, 1e-10, 5000, phi, res, np.zeros(1))
        assert st["status"] == OK and np.array_equal(res, ref[1])
        assert abs(st["iters"][0] - int(ref[3][0])) <= 2
        assert np.linalg.norm(phi - ref[0]) <= 1e-8 * np.linalg.norm(ref[0])
        return st["graph_launches"]
    try:
        gpu.selftest_fail_launch(1, too_large)
        assert (solve() == 0) == bool(persistent)
        gpu.selftest_fail_launch(0)
        assert (solve() == 0) == bool(persistent)  # not tried again on this structure
        gpu.matrix_set(A)
        assert solve() == 0
        gpu.selftest_fail_launch(1, OUT_OF_RESOURCES)
        with pytest.raises(SolverError) as e:
            solve()
        assert e.value.code == DEVICE_ERROR
        gpu.selftest_fail_launch(0)
        assert solve() == 0
    finally:
        gpu.selftest_fail_launch(0)
        gpu.set_option(OPT_PERSISTENT, 0)
