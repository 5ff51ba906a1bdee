"""The batched row sweep: strips and bands of many grids from one queue, the rows
that a warp has not begun taken over by others, and the launches that finish a
step count which three does not divide.  Every member has to equal the same grid
stepped alone by the plain one-step kernel, bit for bit (the kernels run the same
IEEE operations on a cell, so there is no tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tws():
    import terrainwatersim_gb300 as t
    t.lib()
    return t


SWEEP = 7
# widths around a strip's 112 output columns and its 128 loaded ones, heights from
# below the least band to several bands; the last has many bands
SIDES = [(3, 5), (111, 16), (112, 17), (113, 40), (128, 1), (225, 33), (64, 200), (500, 333)]


def make(tws, W, H, seed, flux, bound):
    rng = np.random.default_rng(seed)
    p = tws.params_physical(boundary=bound)
    g = tws.Grid(W, H, p, flux)
    b = rng.uniform(0, 30, (H, W)).astype(np.float32)
    d = rng.uniform(0, 8, (H, W)).astype(np.float32)
    d[rng.uniform(size=(H, W)) < 0.3] = 0
    g.upload(b, d)
    r = max(1, min(W, H) // 4)
    g.set_sources([(tws.SOURCE_DISK, W // 2, H // 2, r, 0.01)] if seed % 2 == 0 else
                  [(tws.SOURCE_BRUSH, W / 3, H / 2, 2.0 + r, 0.02),
                   (tws.SOURCE_DISK, W // 4, H // 3, r, 0.01)])
    return g


@pytest.mark.parametrize("flux", ["FLUX_F32", "FLUX_F16"])
@pytest.mark.parametrize("steps", [3, 4, 49, "each"])
def test_matches_each_grid_alone(tws, flux, steps):
    flux = getattr(tws, flux)
    def grids():
        return [make(tws, W, H, i, flux, tws.BOUNDARY_CLOSED if i % 3 else tws.BOUNDARY_OPEN)
                for i, (W, H) in enumerate(SIDES)]
    counts = [steps] * len(SIDES) if steps != "each" else [0, 1, 2, 3, 7, 8, 60, 100]
    members, alone = grids(), grids()
    with tws.Batch(flux) as batch:
        for g in members:
            batch.add(g)
        batch.set_variant(SWEEP)
        batch.step_each(counts)
        batch.sync()
        for g, ref, n in zip(members, alone, counts):
            ref.set_variant(0)
            ref.step(n)
            for name, x, y in zip(("depth", "flux", "velocity"), g.download(), ref.download()):
                np.testing.assert_array_equal(x.view(np.uint8), y.view(np.uint8),
                                              f"{name} {g.width}x{g.height}")
    for g in members + alone:
        g.close()


def test_taken_for_large_batches_only(tws):
    """Three steps a launch from the size on where it is the faster one, unless a
    variant is set."""
    def launches(W, H, variant=None, disks=0):
        with tws.Batch() as batch:
            gs = [tws.Grid(W, H, tws.params_physical())
                  for _ in range(2)]
            for g in gs:
                g.set_sources(tws.rain_disks(3, W, H, 500, 0.01, disks) if disks else [])
                batch.add(g)
            if variant is not None:
                batch.set_variant(variant)
            batch.step(12)
            batch.sync()
            before = tws.lib().tws_launch_count()
            batch.step(12)
            batch.sync()
            n = tws.lib().tws_launch_count() - before
        for g in gs:
            g.close()
        return n
    assert launches(512, 512) == 6
    assert launches(4096, 2048) == 4
    assert launches(4096, 2048, variant=4) == 6
    assert launches(4096, 2048, disks=8) == 6  # rain on most units
    assert launches(512, 512, variant=SWEEP) == 4
