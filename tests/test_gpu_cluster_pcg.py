"""The PCG of one thread-block cluster per system (SOLV_OPT_PERSISTENT 1 where
the resident PCG does not fit: more systems than SMs, or an unordered system
too large for its gathers), in its three forms, against the oracle and against
the graphs of step kernels.  A first launch refused as too large for a
cooperative one tells the forms apart: the resident solve goes on without it,
a cluster's ends in DEVICE_ERROR."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from programs_b200.mesh import Mesh, poisson_rhs
from programs_b200.solver import (DEVICE_ERROR, MAXITER, OK, OPT_GRAPH_LOOP, OPT_PERSISTENT,
                                  SolverError)

pytestmark = pytest.mark.gpu
TOO_LARGE = 720  # cudaErrorCooperativeLaunchTooLarge


def _hex(nx, ny, nz, order, seed=0):
    m = Mesh.hex(nx, ny, nz, jitter=0.15, seed=seed, permute=True)
    if order:
        m.renumber(order)
    return m.pressure(pin=1)


def _rel(a, b):
    return float(np.linalg.norm(np.ravel(a) - np.ravel(b)) / np.linalg.norm(np.ravel(b)))


def _many(biggest, order, small):
    return [_hex(2 + k % small, 2, 2 + k % small, order, k) for k in range(148)] + [
        _hex(*biggest, order)]


CASES = {
    # at most 1024 and at most 2048 cells a block of 8, in registers and shared memory
    "one_cell_a_thread": lambda: _many((18, 19, 20), Mesh.RCM, 4),
    "two_cells_a_thread": lambda: _many((23, 24, 25), Mesh.RCM, 4),
    # neighbours in other blocks: vectors in global memory, clusters of 8 and of 16
    "unordered": lambda: _many((18, 19, 20), None, 1),
    "unordered_alone": lambda: [_hex(68, 69, 70, None)],
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_cluster_forms(gpu, name):
    mats = CASES[name]()
    cp = gpu.matrix_set_batch(mats)
    b = np.concatenate([poisson_rhs(A.n_cell, 9 + k) for k, A in enumerate(mats)])
    check = sorted({0, len(mats) // 2, len(mats) - 1})
    caps = (3,) if name == "unordered_alone" else (3, 3000)
    refs = {(n, k): Oracle.from_matrix(mats[k]).solv_cg(
        0, 1e-10, n, np.zeros((mats[k].n_cell, 1)), b[cp[k]:cp[k + 1]].reshape(-1, 1))
        for n in caps for k in check}

    def solve(n_iter):
        phi = np.zeros((cp[-1], 1))
        res = np.asfortranarray(b.reshape(-1, 1).copy())
        return phi, gpu.solv_cg_batch(0, 1e-10, n_iter, phi, res)
    try:
        gpu.set_option(OPT_PERSISTENT, 1)
        gpu.selftest_fail_launch(1, TOO_LARGE)
        with pytest.raises(SolverError) as e:
            solve(3)
        assert e.value.code == DEVICE_ERROR
        gpu.selftest_fail_launch(0)
        for n_iter in caps:
            gpu.set_option(OPT_PERSISTENT, 1)
            phi, st = solve(n_iter)
            assert st["graph_launches"] == 0 and st["status"] == (MAXITER if n_iter == 3 else OK)
            for k in check:
                ref = refs[n_iter, k]
                assert abs(int(st["iters_all"][k, 0]) - int(ref[3][0])) <= (0 if n_iter == 3 else 2)
                assert _rel(phi[cp[k]:cp[k + 1]], ref[0]) <= (1e-11 if n_iter == 3 else 1e-8)
            gpu.set_option(OPT_PERSISTENT, 0)
            gpu.set_option(OPT_GRAPH_LOOP, 0)
            phi_g, st_g = solve(n_iter)
            assert st_g["graph_launches"] > 0
            assert np.abs(st_g["iters_all"] - st["iters_all"]).max() <= (0 if n_iter == 3 else 2)
            assert _rel(phi_g, phi) <= (1e-11 if n_iter == 3 else 1e-8)
    finally:
        gpu.selftest_fail_launch(0)
        gpu.set_option(OPT_PERSISTENT, 0)
        gpu.set_option(OPT_GRAPH_LOOP, 2)
