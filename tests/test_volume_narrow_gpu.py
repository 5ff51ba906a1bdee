"""tws_volume on tall grids, whose narrow rows a block sums side by side."""
from __future__ import annotations

import math
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tws():
    import terrainwatersim_gb300 as t
    t.lib()
    return t


@pytest.mark.parametrize("W,H", [(1, 1025), (1, 5000), (3, 2500), (4, 1030), (5, 4097), (8, 20000),
                                 (20, 16384), (127, 1100), (128, 9000), (511, 1500), (512, 1030),
                                 (513, 1030), (1023, 1100), (1025, 1100), (33, 1024)])
@pytest.mark.parametrize("wide", [False, True])
def test_volume_is_the_sum(tws, W, H, wide):
    rng = np.random.default_rng(W + H)
    d = rng.uniform(0.5, 1.0, (H, W))
    d = d * 2.0 ** rng.integers(-60, 60, (H, W)) if wide else np.where(d < 0.7, 0.0, 20.0 * d)
    d = d.astype(np.float32)
    exact = math.fsum(d.ravel().tolist())
    with tws.Grid(W, H) as g:
        g.upload(np.zeros((H, W), np.float32), d)
        got = g.volume()
        again = g.volume()
    # a handful of FP64 roundings per partial sum and in the final tree
    assert abs(got - exact) <= 64 * 2.0 ** -53 * exact
    assert got == again


def test_narrow_rows_take_no_longer_than_wide_ones(tws):
    """The same cells, 2.4 million, in rows of 8 and of 1549: the pitch of 32 reads
    four times the bytes, which come from L2 in a few us.  One by one, the rows of 8
    took more than six times the wide ones' time."""
    best = {}
    for W, H in ((8, 300000), (1549, 1549)):
        with tws.Grid(W, H) as g:
            g.generate_scene(1, 40.0, 15.0)
            g.volume()
            times = []
            for _ in range(50):
                t = time.perf_counter()
                g.volume()
                times.append(time.perf_counter() - t)
            best[W] = min(times)
    assert best[8] < 3 * best[1549], best
