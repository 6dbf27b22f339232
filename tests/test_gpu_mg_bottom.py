"""The V-cycle's coarse levels (k_mg_bottom, k_mg_pre_coarse / _post_coarse)
and the coarsest inverse (k_mg_invert) over their shapes: the inverse in one
block (at most 128 cells) and in a cluster, bottoms of one and several levels,
levels above the bottom.  A wrong coarse correction shows as many times the
iterations, a hand-over to plain PCG, or no convergence: the Jacobi-smoothed
V-cycle takes 20-50 iterations to 1e-12 on these systems (plain Jacobi-PCG
60-700), and at 1e-12 both end within 1e-8 of each other."""
import numpy as np
import pytest

from programs_b200.mesh import Mesh, poisson_rhs
from programs_b200.solver import OK, OPT_MG_SMOOTHER

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(8, 9, 8), (12, 13, 11), (19, 20, 21), (27, 26, 25), (41, 40, 43),
                                  (94, 95, 93)])
def test_solve_through_the_bottom(gpu, dims):
    m = Mesh.hex(*dims, jitter=0.15, seed=6, permute=True)
    m.renumber(Mesh.RCM)
    A = m.pressure(pin=1)
    gpu.matrix_set(A)
    sizes = [A.n_cell]
    while sizes[-1] > 256:
        sizes.append(gpu.mg_aggregates(len(sizes), sizes[-1])[1])
    b = poisson_rhs(A.n_cell, 7).reshape(-1, 1)
    gpu.set_option(OPT_MG_SMOOTHER, 0)
    try:
        phi = np.zeros((A.n_cell, 1))
        st = gpu.solv_fcg(1e-12, 1000, phi, np.asfortranarray(b.copy()), np.zeros(1))
    finally:
        gpu.set_option(OPT_MG_SMOOTHER, 1)
    assert st["status"] == OK and st["fallbacks"] == 0 and st["mg_levels"] == len(sizes) - 1
    assert st["iters"][0] <= 80, st["iters"]
    ref = np.zeros((A.n_cell, 1))
    gpu.solv_cg(0, 1e-12, 20000, ref, np.asfortranarray(b.copy()), np.zeros(1))
    assert np.linalg.norm(phi - ref) <= 1e-8 * np.linalg.norm(ref)
