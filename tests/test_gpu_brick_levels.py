"""Sparse clouds, whose trees leave coarse leaves of every lattice edge: the super-bricks (edge >= 64), the
bricks bounded one depth window at a time, the leaves evaluated without a bound (edge 2), and trees too
shallow for some of them, against the oracle, which evaluates every virtual corner."""
import numpy as np
import pytest

from conftest import sphere

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n,depth", [("sphere", 60, 2), ("sphere", 90, 3), ("torus", 300, 4), ("sphere", 250, 7),
                                          ("torus", 900, 8), ("sphere", 1500, 8)])
def test_mesh_matches_oracle(lib_built, oracle_mod, kind, n, depth):
    import poissonrecon_gpu_gb300 as pg
    from poissonrecon_gpu_gb300 import shapes
    xyz, nrm = sphere(n, seed=5) if kind == "sphere" else shapes.torus(n, seed=5)
    o = oracle_mod.Oracle(depth)
    o.set_points(xyz, nrm)
    o.reconstruct()
    g = pg.Reconstructor(depth=depth)
    g.set_points(xyz, nrm)
    g.build_octree()
    g.compute_rhs()
    g.solve()
    g.set("x", o.get("x"))
    g.eval_points()
    g.set("iso", np.float32([o.get("iso")[0]]))
    g.extract_mesh()
    gv, gf = g.mesh()
    ov = (o.get("mesh_v").reshape(-1, 3) * o.get("scale")[0]).astype(np.float32) + o.get("center")
    of = o.get("mesh_f").reshape(-1, 3)
    assert int(g.get("subdivide_roots")[0]) == int(o.get("subdivide_roots")[0])
    assert len(gf) == len(of)
    row = [("", np.float32)] * 9
    if len(of):
        tg = np.sort(gv[gf].reshape(len(gf), 9).view(row).ravel())
        to = np.sort(ov[of].reshape(len(of), 9).astype(np.float32).view(row).ravel())
        assert np.array_equal(tg, to)
    if depth >= 8:
        assert g.stats()["bricks"] > 0 and max(d for d, c in enumerate(g.stats()["roots_per_depth"]) if c) == depth - 1
    g.close()
