"""The density weights (the splat's walk over the groups of depth k = max(maxDepth - 2, 1), then the samples' 27 nodes)
against a 64-bit restatement over the octree's depth-k nodes: the shallowest tree (k = 1), few and many samples per
node, and copies of a few points.

The bound: a quadratic piece's coefficients reach 4^k, so its float value is within 4 * 4^k * 2^-24 of the spline's,
and a product of three values, each at most 3/4, within e = 3 * (3/4)^2 times that.  W(s) = sum_o B_o(s) w_o then
errs by at most sum_o (e w_o + B_o(s) e n_o), n_o the samples around o, beside the sums' rounding, (n_o + 32) 2^-24
relative; the scale to mean 1 errs by at most the largest relative error of a weight."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def spline(u):
    u = np.abs(u)
    return np.where(u < 0.5, 0.75 - u * u, np.where(u < 1.5, 0.5 * (1.5 - u) ** 2, 0.0))


@pytest.mark.parametrize("n,depth,kind", [(40, 2, "volume"), (2000, 3, "volume"), (3000, 6, "sphere"), (5000, 4, "clusters")])
def test_density_weights(lib_built, n, depth, kind):
    import poissonrecon_gpu_gb300 as pg
    rng = np.random.default_rng(n)
    xyz = rng.random((n, 3), dtype=np.float32)
    if kind == "sphere":
        xyz -= 0.5
        xyz /= np.linalg.norm(xyz, axis=1, keepdims=True)
    if kind == "clusters":
        xyz = xyz[np.arange(n) % 7].copy()
    nrm = rng.standard_normal((n, 3)).astype(np.float32)
    r = pg.Reconstructor(depth=depth, density_weights=True)
    r.set_points(xyz, nrm)
    r.build_octree()
    r.compute_rhs()
    r.solve()
    r.eval_points()
    got = r.get("point_weight").astype(np.float64)
    p = r.get("points").astype(np.float64).reshape(-1, 3)
    base, key = r.get("base"), r.get("key")
    k = max(depth - 2, 1)
    keys = np.asarray(key[base[k]:base[k + 1]]).astype(np.uint64) >> np.uint64(3 * (depth - k))
    r.close()
    c = np.zeros((len(keys), 3), np.int64)
    for b in range(k):
        for ax in range(3):
            c[:, ax] |= ((keys >> np.uint64(3 * b + 2 - ax)) & np.uint64(1)).astype(np.int64) << b
    cell = np.floor(p * 2 ** k).astype(np.int64)
    B = np.ones((len(c), len(p)))
    near = np.ones((len(c), len(p)), bool)
    for ax in range(3):
        B *= spline(p[None, :, ax] * 2 ** k - (c[:, None, ax] + 0.5))
        near &= np.abs(cell[None, :, ax] - c[:, None, ax]) <= 1
    B *= near
    w, no = B.sum(1), near.sum(1)
    W = w @ B
    e = 3 * 0.75 ** 2 * 4 * 4.0 ** k * 2.0 ** -24
    rel = (near.T @ (e * w) + (B * (e * no)[:, None]).sum(0)) / W + (no.max() + 32) * 2.0 ** -24
    assert rel.max() < 0.25
    ref = 1.0 / W
    ref *= len(p) / ref.sum()
    assert np.all(np.abs(got / ref - 1) <= 1.5 * (rel + rel.max()))
