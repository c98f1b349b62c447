"""The flexible CG's grid sums when a wait runs out (an arrival that never comes, PRGPU_HOOK_BARRIER_WAIT): every
block leaves the kernel, the call returns PRGPU_ERR_TIMEOUT, and the context solves as before afterwards."""
import os

import numpy as np
import pytest

from conftest import REPO, sphere

pytestmark = pytest.mark.gpu

CHECKPOINT = os.path.join(REPO, "poissonrecon_gpu_gb300", "weights", "lpc_ellipsoids_d9.bin")


@pytest.mark.parametrize("n,depth,polls", [(20_000, 7, 4000), (3000, 5, 1), (60_000, 9, 100)])
@pytest.mark.parametrize("refine", [0, 1])
def test_learned_solve_wait_runs_out(lib_built, n, depth, polls, refine):
    import poissonrecon_gpu_gb300 as pg
    xyz, nrm = sphere(n, seed=depth)
    r = pg.Reconstructor(depth=depth, solve_mode=pg.SOLVE_RELATIVE, cg_tol=1e-6, preconditioner=CHECKPOINT,
                         refine=bool(refine))
    r.set_points(xyz, nrm)
    r.build_octree()
    r.compute_rhs()
    r.solve()
    x0 = r.get("x")
    pg.test_hook(pg.HOOK_BARRIER_WAIT, polls)
    try:
        with pytest.raises(pg.PrgpuError) as ei:
            r.solve()
        assert ei.value.status == 6
    finally:
        pg.test_hook(pg.HOOK_CLEAR)
    r.set_points(xyz, nrm)
    r.build_octree()
    r.compute_rhs()
    r.solve()
    assert np.array_equal(r.get("x"), x0)
    r.close()
