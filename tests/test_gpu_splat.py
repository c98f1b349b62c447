"""The splat over the occupied cells of a sibling group's block: many points per leaf, blocks filled to every one
of their 64 cells, points at the ends of the domain, and the shallowest and deepest trees, bit for bit against
the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,depth,kind", [(4, 2, "volume"), (3000, 2, "volume"), (20000, 4, "volume"), (5000, 6, "corners"),
                                          (4097, 5, "clusters"), (33, 15, "volume")])
def test_vector_field_matches_oracle(lib_built, oracle_mod, n, depth, kind):
    import poissonrecon_gpu_gb300 as pg
    rng = np.random.default_rng(n)
    xyz = rng.random((n, 3), dtype=np.float32)
    if kind == "corners":
        xyz = np.round(xyz) + np.float32(1e-3) * rng.random((n, 3), dtype=np.float32)
    if kind == "clusters":
        xyz = xyz[np.arange(n) % 5].copy()
    nrm = rng.standard_normal((n, 3)).astype(np.float32)
    g = pg.Reconstructor(depth=depth)
    o = oracle_mod.Oracle(depth)
    g.set_points(xyz, nrm)
    o.set_points(xyz, nrm)
    g.build_octree()
    o.build_octree()
    g.compute_rhs()
    o.build_basis(True)
    o.vector_field()
    assert np.array_equal(g.get("vfield"), o.get("vfield"))
    g.close()
