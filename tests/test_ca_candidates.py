"""The candidate pass of the tile schedules (a warp per candidate on short lists, a thread on long ones) against
the CPU oracle: votes among many flows, falls, ponds, both modes, 2D and 3D, and the list lengths on both
sides of the rule."""
import numpy as np
import pytest

from oracle import oracle as O
from tests import cases as C
from volcano_ca_mc_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sweep", [capi.SWEEP_DENSE, capi.SWEEP_ACTIVE_LIST], ids=["dense", "list"])
@pytest.mark.parametrize("case", [(40, 31, 27, "moore", "periodic", "lava", 0.05), (67, 1, 90, "hexagonal", "periodic", "lava", 0.2),
                                  (48, 33, 20, "von_neumann", "absorbing", "lava", 0.3), (33, 30, 1, "moore", "absorbing", "classic", 0.02),
                                  (40, 31, 27, "pentagonal", "absorbing", "classic", 0.01), (128, 64, 48, "moore", "absorbing", "lava", 0.2),
                                  (128, 64, 48, "pentagonal", "periodic", "classic", 0.2)],
                         ids=lambda c: f"{c[0]}x{c[1]}x{c[2]}-{c[3]}-{c[4]}-{c[5]}")
def test_candidates_match_oracle(case, sweep):
    nx, ny, nz, nb, bc, mode, share = case
    p = capi.CaParams(nx, ny, nz, neighborhood=nb, boundary=bc, seed=3 + nx, max_steps=40, eruption_steps=30, erupt_temp=1200.0,
                      solidus_temp=800.0, cooling_ambient=0.75, cooling_lateral=1.5, cooling_fall=0.5, ponding=True, sweep=sweep, mode=mode)
    rng = np.random.default_rng(nx + nz)
    n = nx * ny * nz
    if mode == "lava":
        kind = rng.choice([0, 1, 2, 3], size=n, p=[0.9 - share, 0.05, share, 0.05]).astype(np.uint8)
        heights = C.terrain(nx, ny, nz, 3)
        per = bc == "periodic"
        spill = O.fill_depressions(heights, nx, ny, per and nx > 1, per and ny > 1)
    else:
        kind = np.where(rng.random(n) < share, 2, 0).astype(np.uint8)
        spill = None
    flow = np.where(kind >= 2, rng.integers(1, 13, size=n), 0).astype(np.int32)
    temp = np.where(kind == 2, rng.uniform(801, 830, size=n), 0.0).astype(np.float32)
    if mode == "classic":
        temp[:] = 0.0
    zero = np.zeros(n, np.uint16)
    s = O.CaState(nx, ny, nz, kind, flow, temp, zero, zero)
    ca = capi.LavaCA(p)
    ca.set_state(s.type, s.flow, s.temp, s.solid, s.arrival, spill, [], steps_done=0)
    op, vt = C.oracle_params(p), O.vent_table([])
    for t in range(5):
        s, counts = O.ca_step(op, t, s, spill, vt)
        ca.step()
        assert C.state_diff(s, ca.download()) == "", f"step {t + 1}"
        if O.ca_stop_after(op, t + 1, counts):
            break
    ca.close()
