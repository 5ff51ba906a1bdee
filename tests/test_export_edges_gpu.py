"""The fused export's edges: widths and heights that are not whole quads, pairs or
blocks, both block sizes, buffers at every alignment it accepts, with and
without a flow map; texels past the buffers stay untouched."""
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


@pytest.mark.parametrize("W,H", [(2, 2), (3, 5), (31, 33), (33, 64), (66, 65), (97, 31), (130, 127),
                                 (1025, 771), (1601, 1603), (1664, 1600)])
@pytest.mark.parametrize("rgba_off,flow_off,flow", [(0, 0, True), (4, 2, True), (8, 0, False)])
def test_any_size_and_alignment(tws, oracle, W, H, rgba_off, flow_off, flow):
    import torch
    levels = min(W, H).bit_length() - 1
    n = sum((W >> l) * (H >> l) * 4 for l in range(1, levels + 1))
    with tws.Grid(W, H) as g:
        g.generate_scene(W + H, 40.0, 15.0)
        if min(W, H) > 8:
            g.set_sources(tws.rain_disks(4, W, H, 3, 0.05, 1))
        g.step(3)
        d, _, v = g.download(flux=False)
        b = g.download_terrain()
        rgba = torch.full((rgba_off + 4 * W * H + 8,), 7.0, device="cuda")
        fm = torch.full((flow_off + 2 * W * H + 8,), 7, dtype=torch.int16, device="cuda")
        mips = torch.full((n + 8,), 7.0, device="cuda")
        torch.cuda.synchronize()
        g.export_textures(rgba.data_ptr() + 4 * rgba_off,
                          fm.data_ptr() + 2 * flow_off if flow else None, levels, mips.data_ptr())
        g.sync()
        rgba, fm, mips = rgba.cpu().numpy(), fm.cpu().numpy(), mips.cpu().numpy()
    want_rgba, want_mips = oracle.terrain_mips(b, d, levels)
    end = rgba_off + 4 * W * H
    assert_bitexact(rgba[rgba_off:end].reshape(H, W, 4), want_rgba, "TerrainData")
    assert np.all(rgba[:rgba_off] == 7.0) and np.all(rgba[end:] == 7.0)
    end = flow_off + 2 * W * H
    if flow:
        assert np.array_equal(fm[flow_off:end].view(np.uint16),
                              v.astype(np.float16).view(np.uint16).ravel())
    assert np.all(fm[:flow_off] == 7) and np.all(fm[end:] == 7)
    off = 0
    for lvl, m in enumerate(want_mips, 1):
        assert_bitexact(mips[off:off + m.size].reshape(m.shape), m, f"mip {lvl}")
        off += m.size
    assert np.all(mips[n:] == 7.0)
