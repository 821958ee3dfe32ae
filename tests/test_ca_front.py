"""The ACTIVE schedule (a list of LAVA cells stepped by the front kernels) against the CPU oracle, bit
for bit: every step's planes, counters and stop reason, over sections and 3D spaces, odd sizes, every
neighbourhood and boundary, and lists longer than the block's shared buffers."""
import numpy as np
import pytest

from oracle import oracle as O
from tests import cases as C
from volcano_ca_mc_b200 import capi

pytestmark = pytest.mark.gpu

CASES = [
    # nx, ny, nz, neighborhood, boundary, steps, vents
    (64, 1, 48, "moore", "absorbing", 120, 1),
    (63, 1, 40, "moore", "periodic", 120, 2),
    (100, 1, 33, "von_neumann", "absorbing", 100, 2),
    (70, 1, 40, "hexagonal", "periodic", 100, 2),
    (64, 1, 48, "pentagonal", "absorbing", 100, 1),
    (24, 20, 16, "moore", "absorbing", 60, 2),
    (33, 17, 14, "moore", "periodic", 60, 2),
    (30, 30, 18, "von_neumann", "periodic", 60, 2),
    (40, 24, 20, "pentagonal", "absorbing", 60, 3),
    (65, 9, 21, "pentagonal", "periodic", 50, 2),
    (2, 3, 30, "moore", "periodic", 40, 1),     # a 2-cell periodic axis: the same cell on both sides
    (3, 2, 2, "moore", "absorbing", 10, 1),     # the smallest space
]


def _params(nx, ny, nz, nb, bc, steps, seed, **over):
    p = dict(neighborhood=nb, boundary=bc, seed=seed, max_steps=steps, eruption_steps=steps // 2, erupt_temp=1200.0,
             solidus_temp=800.0, cooling_ambient=2.0, cooling_lateral=4.0, cooling_fall=2.0, ponding=True,
             sweep=capi.SWEEP_ACTIVE)
    p.update(over)
    return capi.CaParams(nx, ny, nz, **p)


def _follow(ca, op, s, spill, vt, t0, steps):
    act, chg = [], []
    for t in range(t0, t0 + steps):
        s, counts = O.ca_step(op, t, s, spill, vt)
        act.append(int(counts[0]))
        chg.append(int(counts[2]))
        stop = O.ca_stop_after(op, t + 1, counts)
        running = ca.step()
        d = C.state_diff(s, ca.download())
        assert d == "", f"step {t + 1}: {d}"
        info = ca.info()
        assert (info.steps, info.stop_reason, info.lava_cells) == (t + 1, stop, act[-1])
        assert running == (stop == 0)
        if stop:
            break
    return act, chg


@pytest.mark.parametrize("ponding", [True, False], ids=["ponding", "dry"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}x{c[1]}x{c[2]}-{c[3]}-{c[4]}")
def test_lava_steps_match_oracle(case, ponding):
    nx, ny, nz, nb, bc, steps, nv = case
    seed = 1000 + nx * 7 + ny * 13 + nz
    p = _params(nx, ny, nz, nb, bc, steps, seed, ponding=ponding)
    heights = C.terrain(nx, ny, nz, seed)
    vents = C.pick_vents(heights, nx, ny, nz, nv, seed)
    per = bc == "periodic"
    spill = O.fill_depressions(heights, nx, ny, per and nx > 1, per and ny > 1)
    s = C.initial_state(nx, ny, nz, heights, vents, p.erupt_temp)
    ca = capi.LavaCA(p)
    ca.apply_terrain(heights)
    ca.place_seeds(vents)
    act, chg = _follow(ca, C.oracle_params(p), s, spill, O.vent_table(vents), 0, steps)
    assert ca.history() == (act, chg)
    ca.close()


def _scattered(nx, ny, nz, seed, lava):
    """A state of scattered ROCK, BASALT and LAVA (share `lava` of the cells) of a dozen flows, each
    LAVA cell with a temperature of its own around the solidus."""
    rng = np.random.default_rng(seed)
    n = nx * ny * nz
    kind = rng.choice([0, 1, 2, 3], size=n, p=[1 - lava - 0.1, 0.05, lava, 0.05]).astype(np.uint8)
    flow = np.where((kind == 2) | (kind == 3), rng.integers(1, 13, size=n), 0).astype(np.int32)
    temp = np.where(kind == 2, rng.uniform(801, 830, size=n), np.where(kind == 3, 700.0, 0.0)).astype(np.float32)
    solid = np.where(kind == 3, rng.integers(1, 20, size=n), 0).astype(np.uint16)
    arrival = np.where(kind >= 2, rng.integers(0, 20, size=n), 0).astype(np.uint16)
    return O.CaState(nx, ny, nz, kind, flow, temp, solid, arrival)


@pytest.mark.parametrize("case", [(40, 31, 27, "moore", "periodic", 0.05), (40, 31, 27, "pentagonal", "absorbing", 0.3),
                                  (67, 1, 90, "hexagonal", "periodic", 0.2), (48, 33, 20, "von_neumann", "periodic", 0.4)],
                         ids=lambda c: f"{c[0]}x{c[1]}x{c[2]}-{c[3]}-{c[4]}")
def test_scattered_states_match_oracle(case):
    """Falls of every depth, ponds, votes among many flows and cells that solidify in every step; the
    run goes on from the uploaded state, first step by step, then to its end."""
    nx, ny, nz, nb, bc, lava = case
    p = _params(nx, ny, nz, nb, bc, 60, 5 + nx, eruption_steps=40, cooling_ambient=0.75, cooling_lateral=1.5, cooling_fall=0.5)
    heights = C.terrain(nx, ny, nz, 3)
    per = bc == "periodic"
    spill = O.fill_depressions(heights, nx, ny, per and nx > 1, per and ny > 1)
    vents = C.pick_vents(heights, nx, ny, nz, 3, 3)
    s = _scattered(nx, ny, nz, 11 + ny, lava)
    ca = capi.LavaCA(p)
    ca.set_state(s.type, s.flow, s.temp, s.solid, s.arrival, spill, vents, steps_done=20)
    op, vt = C.oracle_params(p), O.vent_table(vents)
    s2 = s
    for t in range(20, 60):
        s2, counts = O.ca_step(op, t, s2, spill, vt)
        stop = O.ca_stop_after(op, t + 1, counts)
        if t < 36:
            ca.step()
            d = C.state_diff(s2, ca.download())
            assert d == "", f"step {t + 1}: {d}"
        if stop:
            break
    ca.run()
    assert ca.info().stop_reason == stop and ca.info().steps == t + 1
    assert C.state_diff(s2, ca.download()) == ""
    ca.close()


@pytest.mark.parametrize("n", [1, 255, 256, 257, 512, 513, 37888, 37889, 40000, 40001, 148 * 1024 + 1])
@pytest.mark.parametrize("mode", ["lava", "classic"])
def test_list_lengths_at_the_edges_of_the_launch_shapes(n, mode):
    """Runs from n LAVA cells of a dozen flows, packed so that most votes count many flows: one block, blocks
    with a slot per thread, blocks that stream, and lists that outgrow the launch they started in."""
    nx, ny, nz = (40, 24, 12) if n < 1000 else (80, 64, 48)
    p = _params(nx, ny, nz, "moore", "periodic", 12, 6 + n, eruption_steps=4, mode=mode)
    rng = np.random.default_rng(n)
    cells = 2 * n if mode == "lava" else min(2 * n + 8, nx * ny * nz)
    at = rng.choice(min(cells, nx * ny * nz), size=n, replace=False)
    kind = np.zeros(nx * ny * nz, np.uint8)
    kind[at] = 2
    flow, temp = np.zeros(kind.size, np.int32), np.zeros(kind.size, np.float32)
    flow[at] = rng.integers(1, 13, size=n)
    temp[at] = rng.uniform(805, 840, size=n)
    zero = np.zeros(kind.size, np.uint16)
    s = O.CaState(nx, ny, nz, kind, flow, temp, zero, zero)
    spill = np.zeros(nx * ny, np.int32) if mode == "lava" else None
    ca = capi.LavaCA(p)
    ca.set_state(s.type, s.flow, s.temp, s.solid, s.arrival, spill, [], steps_done=0)
    op, vt = C.oracle_params(p), O.vent_table([])
    for t in range(12):
        s, counts = O.ca_step(op, t, s, spill, vt)
        stop = O.ca_stop_after(op, t + 1, counts)
        if stop:
            break
    ca.run()
    assert (ca.info().steps, ca.info().stop_reason) == (t + 1, stop)
    assert C.state_diff(s, ca.download()) == ""
    ca.close()


def test_more_solidifying_cells_than_a_block_gathers():
    """Most of a 786 000-cell block of LAVA solidifies in one step."""
    nx, ny, nz = 128, 128, 48
    p = _params(nx, ny, nz, "moore", "absorbing", 30, 4, eruption_steps=0, cooling_ambient=20.0)
    s = _scattered(nx, ny, nz, 2, 0.88)
    spill = np.zeros(nx * ny, np.int32)
    ca = capi.LavaCA(p)
    ca.set_state(s.type, s.flow, s.temp, s.solid, s.arrival, spill, [], steps_done=0)
    _follow(ca, C.oracle_params(p), s, spill, O.vent_table([]), 0, 2)
    ca.close()


def test_more_candidates_than_a_block_gathers():
    """3000 scattered classic seeds reach up to 26 cells each in the first step."""
    nx, ny, nz = 64, 64, 40
    p = capi.CaParams(nx, ny, nz, neighborhood="moore", boundary="periodic", mode="classic", seed=8, max_steps=80)
    idx = np.random.default_rng(8).choice(nx * ny * nz, size=3000, replace=False)
    vents = [(int(i % nx), int((i // nx) % ny), int(i // (nx * ny)), k + 1) for k, i in enumerate(idx)]
    s = C.initial_state(nx, ny, nz, None, vents, 0.0, classic=True)
    ca = capi.LavaCA(p)
    ca.place_seeds(vents)
    _follow(ca, C.oracle_params(p), s, None, O.vent_table(vents), 0, 80)
    ca.close()


@pytest.mark.parametrize("case", [(48, 1, 40, "moore", "periodic"), (20, 16, 12, "pentagonal", "absorbing"),
                                  (31, 27, 1, "hexagonal", "absorbing"), (17, 16, 10, "von_neumann", "periodic")])
def test_classic_steps_match_oracle(case):
    nx, ny, nz, nb, bc = case
    p = capi.CaParams(nx, ny, nz, neighborhood=nb, boundary=bc, mode="classic", seed=77 + nx, max_steps=80)
    idx = np.random.default_rng(nx).choice(nx * ny * nz, size=6, replace=False)
    vents = [(int(i % nx), int((i // nx) % ny), int(i // (nx * ny)), k + 1) for k, i in enumerate(idx)]
    s = C.initial_state(nx, ny, nz, None, vents, 0.0, classic=True)
    ca = capi.LavaCA(p)
    ca.place_seeds(vents)
    _follow(ca, C.oracle_params(p), s, None, O.vent_table(vents), 0, 80)
    ca.close()
