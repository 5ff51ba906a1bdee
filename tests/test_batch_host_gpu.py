"""Host time of a batch call that chooses its kernel by size: for many small members
the choice costs little more than none."""
from __future__ import annotations

import time

import pytest

pytestmark = pytest.mark.gpu


def test_choice_by_size_is_cheap_for_many_small_grids():
    """2000 members: with the choice left open a call looks at each member's size
    once, some nanoseconds each.  30 ns a member, 60 us, is allowed; a search over the
    members for every band height takes several times that."""
    import terrainwatersim_gb300 as tws
    members = 2000
    grids = [tws.Grid(16, 16) for _ in range(members)]

    def best(batch):
        times = []
        for _ in range(60):
            t = time.perf_counter()
            batch.step(3)
            times.append(time.perf_counter() - t)
            batch.sync()
        return min(times)

    with tws.Batch() as batch:
        for g in grids:
            batch.add(g)
        open_choice = best(batch)
        batch.set_variant(4)  # what the open choice takes here
        pinned = best(batch)
    for g in grids:
        g.close()
    assert open_choice - pinned < 30e-9 * members, (open_choice, pinned)
