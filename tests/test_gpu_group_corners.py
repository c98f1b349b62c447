"""Corner values by sibling groups, four groups to a warp, of the finest cells and of the leaves above them: group
counts around that, blocks with every neighbour present (a filled volume), cells at the ends of the domain, lone
groups far apart, and the shallowest tree: the mesh bit for bit the oracle's for the same coefficients."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,depth,kind", [(3, 2, "volume"), (2000, 3, "volume"), (6000, 4, "volume"), (300, 6, "ends"),
                                          (40, 9, "volume"), (7, 7, "volume")])
def test_mesh_matches_oracle(lib_built, oracle_mod, n, depth, kind):
    import poissonrecon_gpu_gb300 as pg
    rng = np.random.default_rng(1000 * depth + n)
    xyz = rng.random((n, 3), dtype=np.float32)
    if kind == "ends":
        xyz = np.round(xyz) + np.float32(1e-3) * rng.random((n, 3), dtype=np.float32)
    nrm = rng.standard_normal((n, 3)).astype(np.float32)
    g = pg.Reconstructor(depth=depth)
    o = oracle_mod.Oracle(depth, threads=4)
    for r in (g, o):
        r.set_points(xyz, nrm)
        r.build_octree()
    g.compute_rhs()
    o.build_basis(True)
    o.vector_field()
    o.divergence()
    o.solve(0, 1e-5, 10000)
    g.solve()
    g.set("x", o.get("x"))
    g.eval_points()
    o.point_values()
    g.set("iso", np.float32([o.get("iso")[0]]))
    g.extract_mesh()
    o.marching_cubes()
    gv, gf = g.mesh()
    ov = o.get("mesh_v").reshape(-1, 3) * o.get("scale")[0] + o.get("center")
    of = o.get("mesh_f").reshape(-1, 3)
    assert len(gf) == len(of)
    tg = np.sort(gv[gf].reshape(len(gf), 9).view([("", np.float32)] * 9).ravel())
    to = np.sort(ov[of].reshape(len(of), 9).astype(np.float32).view([("", np.float32)] * 9).ravel())
    assert np.array_equal(tg, to)
    g.close()
