"""GPU parity of the row sweeps where their 128-column strips, row claims and
division can go wrong: widths around one and two strips, heights around a claim
and the halo, tall grids whose rows idle warps take over, depths outside the
range of the packed division, eight sources at once, and non-finite cells."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_bitexact

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tws():
    import terrainwatersim_gb300 as t
    t.lib()
    return t


def sweeps(tws):
    """The first variant of each depth, and the first one with a tail."""
    picks = {}
    for i, v in enumerate(tws.variants()):
        if v[5] == tws.VARIANT_SWEEP:
            picks.setdefault((v[0], tws.variant_tail_rows(i) > 0), i)
    return sorted(picks.values())


def state(W, H, seed):
    rng = np.random.default_rng(seed)
    b = rng.uniform(0, 6, (H, W)).astype(np.float32)
    d = np.maximum(0, rng.uniform(-2, 5, (H, W))).astype(np.float32)
    f = rng.uniform(0, 0.3, (H, W, 4)).astype(np.float32)
    return b, d, f


def gpu(tws, variant, b, d, f, p, sources, steps, flux=0):
    with tws.Grid(b.shape[1], b.shape[0], p, flux) as g:
        g.upload(b, d, f)
        g.set_sources(sources)
        g.set_variant(variant)
        g.step(steps)
        g.sync()
        return g.download() + (g.buffers().flux_scale,)


def check(tws, oracle, b, d, f, p, sources, steps, bound, flux=0):
    ref = None
    for vi in sweeps(tws):
        gd, gf, gv, scale = gpu(tws, vi, b, d, f, p, sources, steps, flux)
        if ref is None:
            od, of, ov = d.copy(), f.copy(), np.zeros(d.shape + (2,), np.float32)
            kf, ka, c = p.as_tuple()
            if flux:
                oracle.quantize_f16(of, scale)
            oracle.step_f32(b.copy(), od, of, ov, kf, ka, c, bound, [tuple(s) for s in sources],
                            nsteps=steps, flux_scale=scale if flux else 0.0)
            ref = (od, of, ov)
        for name, x, y in zip(("depth", "flux", "flow map"), (gd, gf, gv), ref):
            assert_bitexact(x, y, f"{name} variant {vi}")


@pytest.mark.parametrize("W", [1, 3, 8, 111, 112, 113, 119, 120, 121, 125, 128, 224, 226, 343])
@pytest.mark.parametrize("H,boundary,flux", [(5, "open", 0), (20, "closed", 0), (53, "closed", 1)])
def test_strip_and_claim_edges(tws, oracle, W, H, boundary, flux):
    closed = boundary == "closed"
    p = tws.params_physical(boundary=tws.BOUNDARY_CLOSED if closed else tws.BOUNDARY_OPEN)
    b, d, f = state(W, H, 7 * W + H)
    srcs = [(tws.SOURCE_DISK, W // 2, H // 2, 4, 0.05), (tws.SOURCE_BRUSH, W * 0.9, 1.0, 20.0, 0.4)]
    check(tws, oracle, b, d, f, p, srcs, 12,
          oracle.BOUNDARY_CLOSED if closed else oracle.BOUNDARY_OPEN, flux)


@pytest.mark.parametrize("W,H,flux", [(90, 2500, 0), (600, 1500, 1)])
def test_rows_taken_over(tws, oracle, W, H, flux):
    """More warps than bands, and a slow band under rain: most rows are taken
    over by warps whose queue ran empty."""
    p = tws.params_physical(boundary=tws.BOUNDARY_CLOSED)
    b, d, f = state(W, H, W)
    srcs = [(tws.SOURCE_DISK, W // 2, H // 3, 60, 0.02)]
    check(tws, oracle, b, d, f, p, srcs, 24, oracle.BOUNDARY_CLOSED, flux)


def test_depths_outside_the_packed_division(tws, oracle):
    """Outflow scaling with quotients of denormal, tiny, zero, ordinary and
    huge depths side by side."""
    W, H = 260, 70
    rng = np.random.default_rng(3)
    b = (rng.uniform(0, 1, (H, W)) * 10.0 ** rng.integers(-30, 8, (H, W))).astype(np.float32)
    mag = rng.choice([0.0, 1e-44, 1e-38, 1e-32, 7.8e-31, 8.0e-31, 1e-20, 1e-6, 1.0, 1e6, 1e9], (H, W))
    d = (rng.uniform(0.5, 1, (H, W)) * mag).astype(np.float32)
    f = (rng.uniform(0, 1, (H, W, 4)) * 10.0 ** rng.integers(-40, 9, (H, W, 4))).astype(np.float32)
    p = tws.params_physical(boundary=tws.BOUNDARY_CLOSED)
    check(tws, oracle, b, d, f, p, [], 4, oracle.BOUNDARY_CLOSED)


def test_eight_sources_in_order(tws, oracle):
    W, H = 300, 120
    b, d, f = state(W, H, 8)
    p = tws.params_physical(boundary=tws.BOUNDARY_CLOSED)
    srcs = [(tws.SOURCE_DISK, 100 + 9 * k, 60, 30, 0.01 + 0.003 * k) if k % 3 else
            (tws.SOURCE_BRUSH, 118.0, 55.0 + k, 700.0, 0.3) for k in range(8)]
    check(tws, oracle, b, d, f, p, srcs, 12, oracle.BOUNDARY_CLOSED)


def test_non_finite_cells_as_the_plain_kernel(tws):
    """Infinities and NaNs in the state spread as the one-step kernel spreads
    them (bits equal wherever the value is a number)."""
    W, H = 300, 90
    b, d, f = state(W, H, 5)
    b[20, 30], b[40, 200], d[60, 127], d[10, 250] = np.inf, np.nan, np.inf, np.nan
    d[70, 60], f[30, 112, 1], f[50, 113, 0] = -1.0, np.inf, np.nan
    p = tws.params_physical(boundary=tws.BOUNDARY_OPEN)
    want = gpu(tws, 0, b, d, f, p, [], 4)
    for vi in sweeps(tws):
        for x, y in zip(gpu(tws, vi, b, d, f, p, [], 4)[:3], want[:3]):
            nan = np.isnan(y)
            assert np.array_equal(nan, np.isnan(x)), vi
            assert np.array_equal(x[~nan].view(np.uint32), y[~nan].view(np.uint32)), vi


@pytest.mark.parametrize("size,flux", [((2720, 2700), 0), ((4352, 4100), 1)])
def test_default_from_its_smallest_grids(tws, size, flux):
    """The smallest grids that take the three-step sweep unasked (7 Mi cells, FP16
    flux 17 Mi) against the plain one-step kernel, bit for bit."""
    W, H = size
    out = []
    for variant in (-1, 0):
        with tws.Grid(W, H, tws.params_physical(boundary=tws.BOUNDARY_OPEN), flux) as g:
            g.generate_scene(9, 40.0, 15.0)
            g.set_sources(tws.rain_disks(9, W, H, 40, 0.02, 2))
            if variant >= 0:
                g.set_variant(variant)
            n0 = tws.lib().tws_launch_count()
            g.step(6)
            g.sync()
            out.append((tws.lib().tws_launch_count() - n0, *g.download()))
    assert (out[0][0], out[1][0]) == (2, 6)
    for name, x, y in zip(("depth", "flux", "velocity"), out[0][1:], out[1][1:]):
        np.testing.assert_array_equal(x.view(np.uint8), y.view(np.uint8), name)
