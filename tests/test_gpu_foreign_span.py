"""Brick corners that another leaf owns, filled in several spans (PRGPU_HOOK_FOREIGN_SPAN; by itself a second span needs
2^31 such corners): the mesh is the one of a single launch, with spans that end inside a warp, a block and the list."""
import numpy as np
import pytest

from conftest import sphere

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,depth,spans", [(5000, 6, [1000, 4097]), (100_000, 9, [1 << 17, 300_001, 1 << 40]),
                                           (30_000, 10, [250_000])])
def test_spans_fill_the_same_corners(lib_built, n, depth, spans):
    import poissonrecon_gpu_gb300 as pg
    xyz, nrm = sphere(n, seed=depth)
    g = pg.Reconstructor(depth=depth)
    v0, f0 = g.reconstruct(xyz, nrm)
    before = g.stats()
    assert before["foreign_corners"] > 0 and before["foreign_evaluated"] > 0
    for span in spans:
        pg.test_hook(pg.HOOK_FOREIGN_SPAN, span)
        try:
            v, f = g.reconstruct(xyz, nrm)
        finally:
            pg.test_hook(pg.HOOK_CLEAR)
        assert np.array_equal(v, v0) and np.array_equal(f, f0)
        after = g.stats()
        for k in ("foreign_corners", "foreign_evaluated"):
            assert after[k] == before[k]
    g.close()


def test_span_hook_argument_is_checked(lib_built):
    import poissonrecon_gpu_gb300 as pg
    assert pg._lib().prgpu_test_hook(pg.HOOK_FOREIGN_SPAN, 0, None) == 1
