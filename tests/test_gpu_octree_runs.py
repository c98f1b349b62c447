"""The octree's runs of all depths in one pass: point counts around its tiles of 1,024, many points per leaf
(equal keys across tile ends), one run per depth, and the shallowest and deepest trees, against the oracle."""
import numpy as np
import pytest

from conftest import sphere

pytestmark = pytest.mark.gpu

FIELDS = ("key", "pidx", "pnum", "parent", "children", "neighs", "didx", "dnum", "point_node", "base", "count")


@pytest.mark.parametrize("n,depth,kind", [(2, 2, "sphere"), (31, 15, "sphere"), (1023, 6, "sphere"), (1024, 6, "sphere"),
                                          (1025, 5, "sphere"), (5000, 2, "sphere"), (4097, 9, "clusters"),
                                          (3072, 4, "clusters")])
def test_node_arrays_match_oracle(lib_built, oracle_mod, n, depth, kind):
    import poissonrecon_gpu_gb300 as pg
    xyz, nrm = sphere(n, seed=n)
    if kind == "clusters":      # hundreds of copies of a few points: runs that span tiles
        xyz = xyz[np.arange(n) % 7].copy()
    g = pg.Reconstructor(depth=depth)
    o = oracle_mod.Oracle(depth)
    g.set_points(xyz, nrm)
    o.set_points(xyz, nrm)
    g.build_octree()
    o.build_octree()
    for f in FIELDS:
        assert np.array_equal(g.get(f), o.get(f)), f
    assert np.array_equal(g.get("sort_idx").astype(np.int64), o.get("sort_idx"))
    g.close()
