"""tws_step in a CUDA graph: replays and calls outside the graph in turn carry the
same state on, where the grid's calls outside would take the mesh kernel."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_bitexact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("captured,live", [(4, 8), (4, 4), (8, 40)])
def test_replays_and_live_calls_in_turn(oracle, captured, live):
    import torch
    import terrainwatersim_gb300 as tws
    W, H = 160, 120
    rng = np.random.default_rng(8)
    b = rng.uniform(0, 6, (H, W)).astype(np.float32)
    d = np.maximum(0, rng.uniform(-2, 5, (H, W))).astype(np.float32)
    f = np.zeros((H, W, 4), np.float32)
    p = tws.params_physical(boundary=tws.BOUNDARY_CLOSED)
    stream = torch.cuda.Stream()
    with tws.Grid(W, H, p, stream=stream.cuda_stream) as g:
        g.step(2)  # the kernel is loaded
        g.upload(b, d, f)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            g.step(captured)
        with torch.cuda.stream(stream):
            graph.replay()
            g.step(live)
            graph.replay()
            graph.replay()
            g.step(live)
            graph.replay()
        got = g.download()
    v = np.zeros((H, W, 2), np.float32)
    oracle.step_f32(b, d, f, v, *p.as_tuple(), oracle.BOUNDARY_CLOSED, [],
                    nsteps=4 * captured + 2 * live)
    for name, x, y in zip(("depth", "flux", "flow map"), got, (d, f, v)):
        assert_bitexact(x, y, name)
