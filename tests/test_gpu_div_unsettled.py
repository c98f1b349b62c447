"""The divergence of the two finest depths where three floats do not settle the double sum's rounding and the sum is
formed in double: clouds in which that happens at a node of depth D, of depth D - 1 or of both (one node in 10^5,
found by counting them), and normals that are not numbers, which send every node near them there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cloud(seed, nan, n=20_000):
    rng = np.random.default_rng(seed)
    d = rng.standard_normal((n, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    xyz, nrm = (0.5 + 0.35 * d).astype(np.float32), d.astype(np.float32)
    k = n // 2                          # half the points again, most with the normal turned round
    xyz[k:], nrm[k:] = xyz[:n - k], -nrm[:n - k]
    nrm[k:k + k // 4] = nrm[:k // 4]
    if nan:
        nrm[::997] = np.nan
    return xyz, nrm


@pytest.mark.parametrize("seed,nan", [(2, False), (5, False), (6, False), (5, True)])
def test_fine_divergence_matches_the_double_sums(lib_built, oracle_mod, seed, nan):
    import poissonrecon_gpu_gb300 as pg
    depth = 7
    xyz, nrm = _cloud(seed, nan)
    g = pg.Reconstructor(depth=depth)
    o = oracle_mod.Oracle(depth, threads=4)
    g.set_points(xyz, nrm)
    o.set_points(xyz, nrm)
    g.build_octree()
    o.build_octree()
    g.compute_rhs()
    o.build_basis(True)
    o.vector_field()
    o.divergence()
    base = o.get("base")
    fine = slice(base[depth - 1], base[depth + 1])
    assert np.array_equal(g.get("vfield"), o.get("vfield"), equal_nan=True)
    a, b = g.get("divergence")[fine], o.get("divergence")[fine]
    assert np.array_equal(a, b, equal_nan=True) and np.isnan(a).any() == nan
    g.close()
