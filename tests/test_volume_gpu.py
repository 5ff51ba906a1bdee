"""tws_volume's exact integer sums: depths over the whole range of floats (inside and
outside the integer accumulators), signs, odd widths, unaligned buffers, long
rows, against the correctly rounded sum."""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tws():
    import terrainwatersim_gb300 as t
    t.lib()
    return t


def depths(kind, W, H):
    rng = np.random.default_rng(W + H)
    u = rng.uniform(0.5, 1.0, (H, W))
    if kind == "usual":
        d = np.where(rng.random((H, W)) < 0.6, 0.0, 20.0 * u)
    elif kind == "wide":
        d = u * 2.0 ** rng.integers(-40, 40, (H, W))
    elif kind == "extreme":
        d = u * 2.0 ** rng.integers(-148, 120, (H, W))
    else:
        d = u * 30.0 * rng.choice([-1.0, 1.0], (H, W))
    return d.astype(np.float32)


@pytest.mark.parametrize("kind", ["usual", "wide", "extreme", "signed"])
@pytest.mark.parametrize("W,H", [(1, 1), (5, 3), (255, 130), (1030, 1100), (70000, 2)])
def test_volume_is_the_sum(tws, kind, W, H):
    d = depths(kind, W, H)
    exact = math.fsum(d.ravel().tolist())
    size = math.fsum(np.abs(d.astype(np.float64)).ravel().tolist())
    with tws.Grid(W, H) as g:
        g.upload(np.zeros((H, W), np.float32), d)
        got = g.volume()
    # a handful of FP64 roundings per partial sum and in the final tree
    assert abs(got - exact) <= 64 * 2.0 ** -53 * size


def test_non_finite_depths(tws):
    for bad in (np.inf, np.nan):
        d = np.ones((7, 300), np.float32)
        d[3, 201] = bad
        with tws.Grid(300, 7) as g:
            g.upload(np.zeros_like(d), d)
            got = g.volume()
        assert got == np.inf if bad == np.inf else math.isnan(got)


@pytest.mark.parametrize("offset,pitch", [(0, 333), (1, 340), (4, 336)])
def test_noalloc_takes_any_alignment(tws, offset, pitch):
    import torch
    W, H = 331, 40
    d = depths("wide", W, H)
    buf = torch.full((offset + pitch * H,), 1e9, dtype=torch.float32)
    buf[offset:].view(H, pitch)[:, :W] = torch.from_numpy(d)
    buf = buf.cuda()
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    rc = tws.lib().tws_volume_noalloc(C.c_void_p(buf.data_ptr() + 4 * offset), W, H, pitch, 1.0,
                                      C.c_void_p(out.data_ptr()), None)
    torch.cuda.synchronize()
    exact = math.fsum(d.ravel().tolist())
    assert rc == tws.TWS_OK and abs(out.item() - exact) <= 64 * 2.0 ** -53 * exact
