"""The autotuner where the solve itself would run as one launch (resident
PCG, small systems): it must time the step kernels its settings are for.  The
one-launch kernels take a half or a third of the time of an iteration and do
not know the settings, so the time it reports for the settings before tuning
has to be the step kernels' own, as with GRAPH_LOOP 0, and the solve afterwards
has to run in the form it had."""
import numpy as np
import pytest

from programs_b200.mesh import Mesh, uniform
from programs_b200.solver import (OPT_BLOCK, OPT_GRAPH_ITERS, OPT_GRAPH_LOOP, OPT_GRID_PER_SM,
                                  OPT_PERSISTENT)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,imat,n,persistent", [("cg", 0, 32, 0), ("cg", 0, 32, 1),
                                                    ("cg", 1, 14, 0), ("bicg", 2, 14, 0)])
def test_the_step_kernels_are_timed(gpu, kind, imat, n, persistent):
    m = Mesh.hex(n, jitter=0.15, seed=2, permute=True)
    m.renumber(Mesh.RCM)
    A = m.momentum()[0] if kind == "bicg" else m.pressure(pin=1)
    gpu.matrix_set(A)
    b = uniform(3, A.n_cell).reshape(-1, 1)
    before = {}
    try:
        for loop in (0, 2):
            for k, v in ((OPT_BLOCK, 256), (OPT_GRID_PER_SM, 8), (OPT_GRAPH_ITERS, 16),
                         (OPT_GRAPH_LOOP, loop), (OPT_PERSISTENT, persistent if loop else 0)):
                gpu.set_option(k, v)
            t = gpu.autotune(kind, imat, 1)
            assert t["candidates"] == 10 and 0 < t["ms_per_iter"] <= t["ms_per_iter_before"]
            before[loop] = t["ms_per_iter_before"]
        phi = np.zeros(b.shape)
        st = getattr(gpu, "solv_" + kind)(imat, 1e-6, 200, phi, np.asfortranarray(b.copy()),
                                          np.zeros(1))
    finally:
        for k, v in ((OPT_BLOCK, 256), (OPT_GRID_PER_SM, 8), (OPT_GRAPH_ITERS, 16),
                     (OPT_GRAPH_LOOP, 2), (OPT_PERSISTENT, 0)):
            gpu.set_option(k, v)
    assert 0.7 <= before[2] / before[0] <= 1.4, before
    assert st["graph_launches"] == 0  # one launch, as before
