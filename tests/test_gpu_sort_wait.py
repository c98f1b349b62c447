"""The radix sort whose tiles stop waiting for the tiles before them (PRGPU_HOOK_SORT_POLLS): at once (0), so that every
tile but the first counts the earlier tiles' keys, or after the first look without news (1), so that some do, beside
others that found them.  The order is the oracle's stable one, and the mesh the one of a sort that waits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cloud(n, kind):
    rng = np.random.default_rng(n)
    xyz = rng.random((n, 3), dtype=np.float32)
    if kind == "few":                   # nearly all keys equal: every element of a tile one digit
        xyz[9:] = xyz[rng.integers(0, 9, n - 9)]
    return xyz, rng.standard_normal((n, 3)).astype(np.float32)


@pytest.mark.parametrize("polls", [0, 1])
@pytest.mark.parametrize("n,depth,kind", [(4096, 15, "volume"), (4097, 6, "volume"), (70_001, 9, "few"), (300_007, 11, "volume")])
def test_stable_order_without_waiting(lib_built, oracle_mod, n, depth, kind, polls):
    import poissonrecon_gpu_gb300 as pg
    xyz, nrm = _cloud(n, kind)
    g = pg.Reconstructor(depth=depth)
    o = oracle_mod.Oracle(depth)
    g.set_points(xyz, nrm)
    o.set_points(xyz, nrm)
    pg.test_hook(pg.HOOK_SORT_POLLS, polls)
    try:
        g.build_octree()
    finally:
        pg.test_hook(pg.HOOK_CLEAR)
    o.build_octree()
    assert np.array_equal(g.get("sort_idx").astype(np.int64), o.get("sort_idx"))
    assert np.array_equal(g.get("points"), o.get("points"))
    g.close()


@pytest.mark.parametrize("polls", [0, 1])
def test_mesh_without_waiting(lib_built, polls):
    import poissonrecon_gpu_gb300 as pg
    from conftest import sphere
    xyz, nrm = sphere(100_000, seed=5)
    g = pg.Reconstructor(depth=9)
    v0, f0 = g.reconstruct(xyz, nrm)
    pg.test_hook(pg.HOOK_SORT_POLLS, polls)
    try:
        v, f = g.reconstruct(xyz, nrm)
    finally:
        pg.test_hook(pg.HOOK_CLEAR)
    assert np.array_equal(v, v0) and np.array_equal(f, f0)
    g.close()


def test_sort_hook_argument_is_checked(lib_built):
    import poissonrecon_gpu_gb300 as pg
    assert pg._lib().prgpu_test_hook(pg.HOOK_SORT_POLLS, -1, None) == 1
