"""Batch members whose lists outgrow their blocks within a round (one block, then a slot per thread, then lists
that the blocks stream) against the same jobs alone; a round is 16 steps of every member however its launches
are split."""
import numpy as np
import pytest

from tests import cases as C
from volcano_ca_mc_b200 import capi

pytestmark = pytest.mark.gpu


def _member(kind, k):
    if kind == "classic":  # fills its space: past 592 blocks of 256 slots
        p = capi.CaParams(60, 60, 60, neighborhood="moore", boundary="periodic", mode="classic", seed=k, max_steps=90)
        vents = [(10 + k, 20, 30, 1), (40, 45, 15, 2)]
        heights = None
    elif kind == "fast":
        p = capi.CaParams(70, 64, 40, neighborhood="pentagonal", boundary="absorbing", seed=k, max_steps=70, eruption_steps=60,
                          cooling_ambient=0.5, sweep=capi.SWEEP_ACTIVE)
    else:
        p = capi.CaParams(120, 1, 60, neighborhood="moore", boundary="absorbing", seed=k, max_steps=100, eruption_steps=50,
                          sweep=capi.SWEEP_ACTIVE)
    if kind != "classic":
        heights = C.terrain(p.nx, p.ny, p.nz, k)
        vents = C.pick_vents(heights, p.nx, p.ny, p.nz, 3, k)
    ca = capi.LavaCA(p)
    if heights is not None:
        ca.apply_terrain(heights)
    ca.place_seeds(vents)
    return ca


@pytest.mark.parametrize("kinds", [("classic",), ("fast", "section"), ("section", "classic", "fast", "fast", "section")],
                         ids=lambda k: "-".join(k))
def test_growing_members_match_alone(kinds):
    alone = []
    for k, kind in enumerate(kinds):
        ca = _member(kind, k)
        ca.run()
        alone.append((ca.info().steps, ca.info().stop_reason, ca.history(), ca.download()))
        ca.close()
    batch = capi.CaBatch()
    members = [_member(kind, k) for k, kind in enumerate(kinds)]
    for m in members:
        batch.add(m)
    first, _ = batch.advance(max_graphs=1)
    assert first == []
    batch.remove(members[0])
    assert members[0].info().steps == 16
    batch.add(members[0])
    batch.run()
    for m, (steps, stop, history, state) in zip(members, alone):
        assert (m.info().steps, m.info().stop_reason) == (steps, stop)
        assert m.history() == history
        assert all(np.array_equal(a, b) for a, b in zip(state, m.download()))
        m.close()
    batch.close()
