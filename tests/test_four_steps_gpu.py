"""Calls whose steps leave four over where the library chose the three-step sweep: the
results, and that four steps cost no more than in the two-step tiles, as which
they go."""
from __future__ import annotations

import pytest

from conftest import assert_bitexact

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tws():
    import terrainwatersim_gb300 as t
    t.lib()
    return t


def make(tws, W, H, flux, variant):
    g = tws.Grid(W, H, None, flux)
    g.generate_scene(3, 40.0, 15.0)
    g.set_sources(tws.rain_disks(3, W, H, min(W, H) // 16, 0.01, 8))
    g.set_variant(variant)
    return g


@pytest.mark.parametrize("W,H,flux", [(2720, 2720, 0), (2000, 3701, 0), (4200, 4300, 1)])
@pytest.mark.parametrize("steps", [4, 7])
def test_as_the_plain_kernel(tws, W, H, flux, steps):
    out = []
    for variant in (-1, 0):
        with make(tws, W, H, flux, variant) as g:
            if variant < 0:
                assert tws.variants()[g.current_variant()][5] == tws.VARIANT_SWEEP
            n0 = tws.lib().tws_launch_count()
            g.step(steps)
            if variant < 0:
                assert tws.lib().tws_launch_count() - n0 == (steps + 2) // 3
            out.append(g.download())
    for name, x, y in zip(("depth", "flux", "flow map"), *out):
        assert_bitexact(x, y, name)


def test_four_steps_take_no_longer_than_as_tiles(tws):
    """The same two launches; a tenth is allowed for noise (three and one take a
    fifth more)."""
    import torch
    best = {}
    for variant in (-1, 16):
        with make(tws, 2720, 2720, 0, variant) as g:
            stream = torch.cuda.ExternalStream(g.stream)
            g.step(4)
            times = []
            for _ in range(12):
                a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                a.record(stream)
                for _ in range(5):
                    g.step(4)
                b.record(stream)
                g.sync()
                times.append(a.elapsed_time(b))
            best[variant] = min(times)
    assert best[-1] < 1.1 * best[16], best
