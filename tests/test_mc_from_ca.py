"""Domain and cooling mobility taken from a CA handle on the device (CoolingMobility,
engine/src/mc/CoolingMobility.cpp:8-83) against the oracle, for rows of each group width (16, 4 and 1
cells per thread), and the colour lists a whole space builds only when they are asked for."""
import numpy as np
import pytest

from oracle import oracle as O
from tests import cases as C
from volcano_ca_mc_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(48, 20, 16), (44, 18, 15), (33, 17, 14), (70, 1, 37), (512, 1, 48)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("steps", [3, 60])
def test_domain_and_mobility_from_ca(shape, steps):
    nx, ny, nz = shape
    p = capi.CaParams(nx, ny, nz, neighborhood="moore", boundary="absorbing", seed=4, max_steps=steps, eruption_steps=20,
                      cooling_ambient=12.0, cooling_lateral=20.0, cooling_fall=2.0)
    heights = C.terrain(nx, ny, nz, 4)
    vents = C.pick_vents(heights, nx, ny, nz, 2, 4)
    ca = capi.LavaCA(p)
    ca.apply_terrain(heights)
    ca.place_seeds(vents)
    ca.run()
    s = O.CaState(nx, ny, nz, *ca.download())
    domain = O.basalt_domain(s)
    mob = O.mobility_from_cooling(s, domain, 0.05)
    mc = capi.PottsMC(capi.McParams(nx, ny, nz, neighborhood="moore", seed=2, Q=30, kT=0.5))
    mc.set_domain_from_ca(ca)
    for _ in range(2):
        mc.set_mobility_from_ca(ca, 0.05, True)
        assert np.array_equal(mc.mobility().view(np.uint32), mob.astype(np.float32).view(np.uint32))
    mc.initialize()
    mp = O.mc_params(nx, ny, nz, "moore", "absorbing", False, 2, 30, 1.0, 0.5)
    spin = O.mc_init(mp, domain)
    assert np.array_equal(mc.crystals(), spin) and mc.info().domain_cells == int(domain.sum())
    for t in range(2):
        O.mc_sweep(mp, t, domain, mob, spin)
    mc.sweep(2)
    assert np.array_equal(mc.crystals(), spin)
    mc.close()
    ca.close()


@pytest.mark.parametrize("case", [("moore", (14, 11, 9)), ("von_neumann", (12, 10, 8))])
def test_colour_passes_after_whole_space_sweeps(case):
    nb, (nx, ny, nz) = case
    domain = np.ones(nx * ny * nz, np.uint8)
    mp = O.mc_params(nx, ny, nz, nb, "periodic", True, 6, 25, 1.0, 0.5)
    spin = O.mc_init(mp, domain)
    mc = capi.PottsMC(capi.McParams(nx, ny, nz, neighborhood=nb, boundary="periodic", domain_full=True, seed=6, Q=25, kT=0.5))
    mc.set_domain(None)
    mc.initialize()
    info = mc.info()
    assert info.domain_cells == nx * ny * nz and info.colors == O.mc_colors(mp)
    mc.sweep(2)
    for c in range(info.colors):
        mc.color_pass(c)
    mc.sweep(1)
    for t in range(4):
        O.mc_sweep(mp, t, domain, None, spin)
    assert np.array_equal(mc.crystals(), spin)
    assert mc.energy() == O.mc_energy(mp, 4, spin) and mc.info().sweeps == 4
    mc.close()
