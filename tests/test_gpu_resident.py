"""The resident FP64 Jacobi PCG (k_pcg_grid: the library's own choice for
systems that fit the SMs) at the edges of its shapes, against the oracle.
Per-cell arithmetic is the step kernels', so the bars are the parity tests':
the initial residual bit for bit, iteration counts within 2, solutions
within 1e-8 at a 1e-10 residual; a capped solve differs by the summation
order of the reductions alone (a few 1e-16 per step): 1e-11 after 3."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from programs_b200.mesh import FaceMatrix, Mesh, poisson_rhs
from programs_b200.solver import MAXITER, OK

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm(np.ravel(a) - np.ravel(b)) / np.linalg.norm(np.ravel(b)))


def _hex(nx, ny, nz, order=Mesh.RCM, seed=0):
    m = Mesh.hex(nx, ny, nz, jitter=0.15, seed=seed, permute=True)
    if order:
        m.renumber(order)
    return m.pressure(pin=1)


def _wide(n, per, seed):
    """Rows of up to 30 slots and more, so only part of them fits shared memory."""
    rng = np.random.default_rng(seed)
    pairs = sorted({(int(a), k) for k in range(2, n + 1)
                    for a in rng.integers(max(1, k - 400), k, per)})
    ip, inb = (np.array(c, np.int32) for c in zip(*pairs))
    p = -rng.uniform(0.2, 1.0, len(ip))
    pl = 1.0 - np.bincount(ip - 1, p, n) - np.bincount(inb - 1, p, n)
    return FaceMatrix(n, ip, inb, p, p.copy(), pl)


CASES = {  # cells: one block; two ragged ones; a full wave; 2, 3 and 4 cells a thread
    "1x1x3": lambda: _hex(1, 1, 3, None),
    "8x8x8": lambda: _hex(8, 8, 8),
    "8x9x8": lambda: _hex(8, 9, 8),
    "41x43x43": lambda: _hex(41, 43, 43),
    "63x64x67_none": lambda: _hex(63, 64, 67, None),
    "71x70x73": lambda: _hex(71, 70, 73),
    "71x70x73_none": lambda: _hex(71, 70, 73, None),
    "80x81x79": lambda: _hex(80, 81, 79),
    "wide": lambda: _wide(60000, 15, 3),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_capped_and_full_solves(gpu, name):
    A = CASES[name]()
    gpu.matrix_set(A)
    o = Oracle.from_matrix(A)
    N = A.n_cell
    b = poisson_rhs(N, 4).reshape(-1, 1)
    full = N < 100000 or name == "wide"
    for reduc, n_iter in [(1e-30, 3)] + [(1e-10, 5000)] * full:
        ref = o.solv_cg(0, reduc, n_iter, np.zeros((N, 1)), b)
        phi, res0, rn = np.zeros((N, 1)), np.asfortranarray(b.copy()), np.zeros(1)
        st = gpu.solv_cg(0, reduc, n_iter, phi, res0, rn)
        assert np.array_equal(res0, ref[1])
        if n_iter == 3 and N > 3:
            assert st["status"] == MAXITER and st["iters"][0] == 3
            assert _rel(phi, ref[0]) <= 1e-11
        elif n_iter > 3:
            assert st["status"] == OK and abs(st["iters"][0] - int(ref[3][0])) <= 2
            assert _rel(phi, ref[0]) <= 1e-8


@pytest.mark.parametrize("n_sys", [3, 149])  # 149: more systems than SMs, the step kernels
def test_uneven_batch(gpu, n_sys):
    mats = [_hex(3 + k % 5, 4, 3 + k % 7, seed=k) for k in range(n_sys - 1)] + [_hex(20, 21, 22)]
    cp = gpu.matrix_set_batch(mats)
    b = np.concatenate([poisson_rhs(A.n_cell, 9 + k) for k, A in enumerate(mats)])
    for n_iter in (2, 3000):
        phi = np.zeros((cp[-1], 1))
        st = gpu.solv_cg_batch(0, 1e-10, n_iter, phi, np.asfortranarray(b.reshape(-1, 1).copy()))
        assert st["status"] == (OK if n_iter > 2 else MAXITER)
        for k in (0, 1, n_sys - 1):
            sl = slice(cp[k], cp[k + 1])
            ref = Oracle.from_matrix(mats[k]).solv_cg(
                0, 1e-10, n_iter, np.zeros((mats[k].n_cell, 1)), b[sl].reshape(-1, 1))
            assert abs(int(st["iters_all"][k, 0]) - int(ref[3][0])) <= 2
            assert _rel(phi[sl], ref[0]) <= (1e-8 if n_iter > 2 else 1e-11)
