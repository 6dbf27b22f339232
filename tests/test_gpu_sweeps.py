"""The DIC/DILU recurrences (kernels.cuh: sweep_rows) on the structures where
their chunks, their gate and their slices end: rows wider than one chunk of
slots, slices that hold many levels (cells that wait for cells of the same
warp), orders of few levels, several components.  Bit-exact against the
oracle for the factorisation and the sweeps; capped solves, whose only other
difference is the reductions' summation order (a few 1e-16 per step), to
1e-11."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from programs_b200.mesh import FaceMatrix, Mesh, uniform
from programs_b200.solver import MAXITER, OK, OPT_GRAPH_LOOP, ZERO_RHS

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[2, 0], ids=["chosen", "step_kernels"])
def solver(gpu, request):
    gpu.set_option(OPT_GRAPH_LOOP, request.param)
    yield gpu
    gpu.set_option(OPT_GRAPH_LOOP, 2)


def _from_pairs(n, pairs, seed):
    """A diagonally dominant face matrix with the given couplings (1-based)."""
    rng = np.random.default_rng(seed)
    ip, inb = (np.array(c, np.int32) for c in zip(*pairs))
    p, q = -rng.uniform(0.2, 1.0, (2, len(ip)))
    pl = 1.0 - np.bincount(ip - 1, p, n) - np.bincount(inb - 1, q, n)
    return FaceMatrix(n, ip, inb, p, q, pl)


def _chain(n):
    return _from_pairs(n, [(k, k + 1) for k in range(1, n)], 1)


def _random(n, per, seed, swap=False):
    rng = np.random.default_rng(seed)
    pairs = {(int(a), k) for k in range(2, n + 1) for a in rng.integers(1, k, per)}
    pairs = sorted(pairs)
    if swap:  # owner above neighbour: the sweep coefficients differ from the product's
        pairs = [(b, a) if (a + b) % 3 == 0 else (a, b) for a, b in pairs]
    return _from_pairs(n, pairs, seed)


def _hex(nx, ny, nz, order):
    m = Mesh.hex(nx, ny, nz, jitter=0.15, seed=3, permute=True)
    m.renumber(order)
    return m.momentum()[0]


CASES = {
    "chain_70": lambda: _chain(70),
    "chain_9": lambda: _chain(9),
    "narrow_2x2x50": lambda: _hex(2, 2, 50, Mesh.RCM),
    "star_41": lambda: _from_pairs(41, [(1, k) for k in range(2, 42)], 2),
    "random_5": lambda: _random(333, 5, 4),
    "random_13_swapped": lambda: _random(500, 13, 5, swap=True),
    "hex_rcm": lambda: _hex(11, 13, 12, Mesh.RCM),
    "hex_color": lambda: _hex(11, 13, 12, Mesh.COLOR),
    "one_deep": lambda: _hex(37, 21, 1, Mesh.RCM),
}


@pytest.fixture(scope="module", params=sorted(CASES))
def case(request, gpu):
    A = CASES[request.param]()
    gpu.matrix_set(A)
    return A, Oracle.from_matrix(A)


@pytest.mark.parametrize("imat", [1, 2])
def test_factorisation_and_sweeps(gpu, case, imat):
    A, o = case
    c_ref, cr_ref = o.solv_precond(imat)
    c, cr = np.empty(A.n_cell), np.empty(A.n_cell)
    gpu.solv_precond(imat, c, cr)
    assert np.array_equal(cr, cr_ref) and np.array_equal(c, c_ref)
    for seed in (9, 10):  # the second finds the buffers as the first left them
        b = uniform(seed, A.n_cell)
        x = np.zeros(A.n_cell)
        gpu.solv_direct(imat, c, cr, x, b)
        assert np.array_equal(x, o.solv_direct(imat, c_ref, cr_ref, b))


@pytest.mark.parametrize("kind,imat", [("bicg", 2), ("bicg", 0), ("cg", 1), ("cg", 0)])
@pytest.mark.parametrize("V", [1, 2, 3, 4])
@pytest.mark.parametrize("not_r0", [False, True])
def test_capped_solve(solver, case, V, kind, imat, not_r0):
    A, o = case
    phi = uniform(5, A.n_cell * V).reshape(A.n_cell, V).copy()
    b = uniform(6, A.n_cell * V).reshape(V, A.n_cell).T.copy(order="F")
    ref = getattr(o, "solv_" + kind)(imat, 1e-30, 2, phi.copy(), b.copy(order="F"), not_r0)
    rn = np.zeros(V)
    st = getattr(solver, "solv_" + kind)(imat, 1e-30, 2, phi, b, rn, not_r0)
    assert st["status"] == MAXITER and st["iters"] == [2] * V
    assert np.array_equal(b, ref[1]) and np.allclose(rn, ref[2], rtol=1e-12, atol=0)
    assert np.linalg.norm(phi - ref[0]) <= 1e-11 * np.linalg.norm(ref[0])


def test_lanes_that_stop_apart_and_zero_right_hand_sides(solver):
    """Components converge at their own iterations; a zero component beside
    others takes one iteration, as in the reference's loop; all zero is its
    early return, phi untouched."""
    A = _hex(7, 8, 9, Mesh.RCM)
    o = Oracle.from_matrix(A)
    solver.matrix_set(A)
    N = A.n_cell
    b = np.zeros((N, 3), order="F")
    b[:, 0] = uniform(3, N)
    b[5, 2] = 1.0
    for kind, imat in (("bicg", 2), ("cg", 1), ("bicg", 0)):
        ref = getattr(o, "solv_" + kind)(imat, 1e-10, 500, np.zeros((N, 3)), b)
        phi, rn = np.zeros((N, 3)), np.zeros(3)
        st = getattr(solver, "solv_" + kind)(imat, 1e-10, 500, phi, b.copy(order="F"), rn)
        assert st["status"] == (OK if np.all(ref[4] < 1e-10) else MAXITER)
        assert st["iters"][1] == int(ref[3][1])
        for v in range(3):  # where the reference's iteration converges (CG need not here)
            if ref[4][v] < 1e-10:
                assert abs(st["iters"][v] - int(ref[3][v])) <= 2
                assert (np.linalg.norm(phi[:, v] - ref[0][:, v])
                        <= 1e-8 * np.linalg.norm(ref[0][:, v]))
        phi = np.ones((N, 3))
        st = getattr(solver, "solv_" + kind)(imat, 1e-10, 500, phi, np.zeros((N, 3), order="F"),
                                             rn, True)
        assert st["status"] == ZERO_RHS and st["iters"] == [0] * 3 and np.all(phi == 1.0)


@pytest.mark.parametrize("n_sys", [2, 13, 900])  # fewer systems than blocks, and more
def test_batch_of_systems_that_share_slices(solver, n_sys):
    """Systems end inside slices; each must come out as by itself."""
    gpu = solver
    mats = [_hex(2 + k % 3, 3, 2 + k % 5, Mesh.RCM) if k % 4 else _chain(3 + k % 37)
            for k in range(n_sys - 1)] + [_hex(9, 10, 11, Mesh.RCM)]
    cp = gpu.matrix_set_batch(mats)
    b = uniform(4, cp[-1])
    phi = np.zeros((cp[-1], 1))
    gpu.solv_bicg_batch(2, 1e-30, 2, phi, np.asfortranarray(b.reshape(-1, 1).copy()))
    for k in sorted({0, 1, n_sys // 2, n_sys - 2, n_sys - 1}):
        sl = slice(cp[k], cp[k + 1])
        ref = Oracle.from_matrix(mats[k]).solv_bicg(2, 1e-30, 2, np.zeros((mats[k].n_cell, 1)),
                                                    b[sl].reshape(-1, 1))
        assert np.linalg.norm(phi[sl] - ref[0]) <= 1e-11 * np.linalg.norm(ref[0])
    b[: cp[1]] = 0.0  # one system without a right-hand side, then none with one
    phi = np.zeros((cp[-1], 1))
    st = gpu.solv_bicg_batch(2, 1e-10, 200, phi, np.asfortranarray(b.reshape(-1, 1).copy()))
    assert st["status"] == OK and st["iters_all"][0, 0] == 1 and np.all(phi[: cp[1]] == 0.0)
    st = gpu.solv_bicg_batch(2, 1e-10, 200, phi, np.zeros((cp[-1], 1), order="F"), True)
    assert st["status"] == ZERO_RHS and np.all(st["iters_all"] == 0)


@pytest.mark.parametrize("dims,V", [((16, 16, 32), 1), ((16, 17, 32), 1), ((16, 16, 16), 2),
                                    ((13, 14, 15), 3), ((12, 13, 13), 4)])
def test_at_the_small_solve_s_limit(gpu, dims, V):
    """8192 values (cells x components) a system is its last size."""
    A = _hex(*dims, Mesh.RCM)
    o = Oracle.from_matrix(A)
    gpu.matrix_set(A)
    N = A.n_cell
    b = uniform(6, N * V).reshape(V, N).T.copy(order="F")
    ref = o.solv_bicg(2, 1e-10, 100, np.zeros((N, V)), b)
    phi = np.zeros((N, V))
    st = gpu.solv_bicg(2, 1e-10, 100, phi, b.copy(order="F"), np.zeros(V))
    assert st["status"] == OK and all(abs(x - int(y)) <= 2 for x, y in zip(st["iters"], ref[3]))
    assert np.linalg.norm(phi - ref[0]) <= 1e-8 * np.linalg.norm(ref[0])
