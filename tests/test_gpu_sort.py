"""The sort behind the octree around its tiles of 4,096 keys: single tiles, ragged ends, many tiles, keys that
are all or nearly all equal (every element one digit, order kept), and one to six passes (depths 2 to 15),
against the oracle's stable order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,depth,kind", [(2, 2, "volume"), (33, 2, "volume"), (4095, 3, "volume"), (4096, 15, "volume"),
                                          (4097, 6, "volume"), (12_289, 8, "equal"), (40_001, 5, "few"),
                                          (300_007, 9, "few"), (1_000_003, 11, "volume")])
def test_stable_order(lib_built, oracle_mod, n, depth, kind):
    import poissonrecon_gpu_gb300 as pg
    rng = np.random.default_rng(n)
    xyz = rng.random((n, 3), dtype=np.float32)
    if kind != "volume":                # the first points span the cube, the rest are copies
        k = 2 if kind == "equal" else 9
        xyz[k:] = xyz[1 if kind == "equal" else rng.integers(0, k, n - k)]
    nrm = rng.standard_normal((n, 3)).astype(np.float32)
    g = pg.Reconstructor(depth=depth)
    o = oracle_mod.Oracle(depth)
    g.set_points(xyz, nrm)
    o.set_points(xyz, nrm)
    g.build_octree()
    o.build_octree()
    assert np.array_equal(g.get("sort_idx").astype(np.int64), o.get("sort_idx"))
    assert np.array_equal(g.get("points"), o.get("points"))
    g.close()
