"""Tiles whose threads keep pairs of cells in registers: grids that end inside a
pair, on a tile's edge and just past it, rain and a brush across tile borders and
in the corner.  Every result has to equal the plain one-step kernel's, bit for bit
(the same IEEE operations on every cell, so there is no tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tws():
    import terrainwatersim_gb300 as t
    t.lib()
    return t


SIZES = [(1, 1), (2, 33), (31, 32), (33, 31), (64, 65), (95, 97), (129, 70)]


def run(tws, size, flux, bound, variant, batch):
    W, H = size
    rng = np.random.default_rng(W * 1000 + H)
    b = rng.uniform(0, 30, (H, W)).astype(np.float32)
    d = rng.uniform(0, 8, (H, W)).astype(np.float32)
    d[rng.uniform(size=(H, W)) < 0.3] = 0
    f = rng.uniform(0, 0.3, (H, W, 4)).astype(np.float32)
    with tws.Grid(W, H, tws.params_physical(boundary=bound), flux) as g:
        g.upload(b, d, f)
        g.set_sources([(tws.SOURCE_DISK, W // 2, H // 2, max(1, W // 5), 0.05),
                       (tws.SOURCE_BRUSH, W * 0.9, 1.0, 20.0, 0.4),
                       (tws.SOURCE_DISK, W - 1, H - 1, 1, 0.01)])
        if batch:
            with tws.Batch(flux) as many:
                many.add(g)
                many.set_variant(variant)
                many.step(6)
                many.sync()
        else:
            g.set_variant(variant)
            g.step(6)
            g.sync()
        return g.download()


@pytest.mark.parametrize("flux", [0, 1])
@pytest.mark.parametrize("size", SIZES)
def test_equals_the_plain_kernel(tws, size, flux):
    for bound in (tws.BOUNDARY_OPEN, tws.BOUNDARY_CLOSED):
        ref = run(tws, size, flux, bound, 0, False)
        for variant, batch in ((16, False), (18, False), (4, True), (6, True)):
            for name, x, y in zip(("depth", "flux", "velocity"),
                                  run(tws, size, flux, bound, variant, batch), ref):
                np.testing.assert_array_equal(x.view(np.uint8), y.view(np.uint8),
                                              f"{name} variant {variant} batch {batch}")
