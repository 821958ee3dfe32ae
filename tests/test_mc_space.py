"""Whole-space Potts sweeps (four cells of a colour per thread on a byte copy of the orientations)
against the CPU oracle, bit for bit: row lengths around the group of eight, odd wrapped axes (a third
colour class), open frames, every neighbourhood, planes in each orientation, the smallest and largest
Q, and the spaces just past the rule (Q > 256, rows shorter than 6), which take the list sweeps."""
import numpy as np
import pytest

from oracle import oracle as O
from volcano_ca_mc_b200 import capi

pytestmark = pytest.mark.gpu

CASES = [
    # nb, bc, dims, Q, kT, mobility
    *[("moore", "periodic", (nx, 5, 4), 20, 0.7, False) for nx in range(5, 19)],
    *[("von_neumann", "absorbing", (nx, 6, 5), 12, 0.6, False) for nx in (6, 7, 8, 9, 15, 16, 17)],
    ("moore", "absorbing", (15, 7, 9), 2, 0.4, False),
    ("moore", "absorbing", (24, 1, 31), 256, 0.0, True),
    ("moore", "periodic", (257, 2, 3), 3, 0.9, False),
    ("von_neumann", "periodic", (16, 10, 12), 7, 0.0, True),
    ("von_neumann", "periodic", (17, 9, 4), 64, 0.5, True),
    ("pentagonal", "periodic", (23, 13, 11), 40, 0.6, False),
    ("pentagonal", "absorbing", (40, 9, 6), 256, 0.6, True),
    ("pentagonal", "absorbing", (19, 14, 1), 5, 0.5, False),
    ("hexagonal", "periodic", (31, 17, 1), 64, 0.6, True),
    ("hexagonal", "absorbing", (26, 1, 19), 30, 0.3, False),
    ("hexagonal", "periodic", (1, 27, 18), 30, 0.3, True),
    ("moore", "periodic", (1, 21, 35), 50, 0.5, False),
    ("von_neumann", "absorbing", (1, 6, 50), 9, 0.5, False),
    ("moore", "absorbing", (1, 5, 20), 9, 0.5, False),
    ("moore", "periodic", (20, 10, 6), 257, 0.6, False),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}-{c[1]}-{'x'.join(map(str, c[2]))}-Q{c[3]}")
def test_space_sweeps_match_oracle(case):
    nb, bc, (nx, ny, nz), Q, kT, use_mob = case
    seed = 7 + nx + 3 * ny
    n = nx * ny * nz
    domain = np.ones(n, np.uint8)
    mob = np.random.default_rng(seed).uniform(0.2, 1.0, n).astype(np.float32) if use_mob else None
    mp = O.mc_params(nx, ny, nz, nb, bc, True, seed, Q, 1.0, kT)
    spin = O.mc_init(mp, domain)
    mc = capi.PottsMC(capi.McParams(nx, ny, nz, neighborhood=nb, boundary=bc, domain_full=True, seed=seed, Q=Q, kT=kT))
    mc.set_domain(None)
    if use_mob:
        mc.set_mobility(mob)
    mc.initialize()
    assert np.array_equal(mc.crystals(), spin)
    tot = np.zeros(3, np.uint64)
    done = 0
    for count in (1, 3, 2):
        before = int(tot[1])
        for _ in range(count):
            tot += O.mc_sweep(mp, done, domain, mob, spin)
            done += 1
        assert mc.sweep(count) == int(tot[1]) - before
        got = mc.crystals()
        assert np.array_equal(got, spin), f"sweep {done}: {(got != spin).sum()} cells differ"
        assert mc.energy() == O.mc_energy(mp, done, spin)
    info = mc.info()
    assert (info.attempts, info.accepted, info.uphill, info.sweeps) == (*(int(v) for v in tot), done)
    mc.close()


@pytest.mark.parametrize("case", [("moore", "periodic", (6, 5, 4), 20, 0.7, False), ("moore", "periodic", (17, 9, 7), 256, 0.5, True),
                                  ("von_neumann", "periodic", (17, 9, 4), 64, 0.5, True), ("pentagonal", "absorbing", (40, 9, 6), 129, 0.6, True),
                                  ("hexagonal", "periodic", (31, 17, 1), 2, 0.0, False), ("von_neumann", "absorbing", (480, 200, 1), 9, 0.5, False),
                                  ("von_neumann", "absorbing", (480, 201, 1), 9, 0.5, False)],
                         ids=lambda c: f"{c[0]}-{c[1]}-{'x'.join(map(str, c[2]))}-Q{c[3]}")
def test_small_spaces_match_oracle(case):
    """Calls of four and more MCS on small spaces (a cell per thread) and shorter calls before and after them,
    up to the widest colour that is still taken that way and one row beyond."""
    nb, bc, (nx, ny, nz), Q, kT, use_mob = case
    seed = 31 + nx + 3 * ny
    n = nx * ny * nz
    domain = np.ones(n, np.uint8)
    mob = np.random.default_rng(seed).uniform(0.2, 1.0, n).astype(np.float32) if use_mob else None
    mp = O.mc_params(nx, ny, nz, nb, bc, True, seed, Q, 1.0, kT)
    spin = O.mc_init(mp, domain)
    mc = capi.PottsMC(capi.McParams(nx, ny, nz, neighborhood=nb, boundary=bc, domain_full=True, seed=seed, Q=Q, kT=kT))
    mc.set_domain(None)
    if use_mob:
        mc.set_mobility(mob)
    mc.initialize()
    tot = np.zeros(3, np.uint64)
    done = 0
    for count in (1, 4, 2, 5):
        before = int(tot[1])
        for _ in range(count):
            tot += O.mc_sweep(mp, done, domain, mob, spin)
            done += 1
        assert mc.sweep(count) == int(tot[1]) - before
        got = mc.crystals()
        assert np.array_equal(got, spin), f"sweep {done}: {(got != spin).sum()} cells differ"
        assert mc.energy() == O.mc_energy(mp, done, spin)
    info = mc.info()
    assert (info.attempts, info.accepted, info.uphill, info.sweeps) == (*(int(v) for v in tot), done)
    mc.close()


@pytest.mark.parametrize("dims", [(128, 95, 98), (128, 96, 99), (300, 160, 51)], ids=lambda d: "x".join(map(str, d)))
def test_space_block_sizes_match_oracle(dims):
    """Spaces below, at and above a group of eight cells per thread of the large blocks (148 x 512 groups a colour)."""
    nx, ny, nz = dims
    n = nx * ny * nz
    domain = np.ones(n, np.uint8)
    for nb, Q in (("moore", 200), ("von_neumann", 20)):
        mp = O.mc_params(nx, ny, nz, nb, "absorbing", True, 5, Q, 1.0, 0.6)
        spin = O.mc_init(mp, domain)
        mc = capi.PottsMC(capi.McParams(nx, ny, nz, neighborhood=nb, boundary="absorbing", domain_full=True, seed=5, Q=Q, kT=0.6))
        mc.set_domain(None)
        mc.initialize()
        tot = np.zeros(3, np.uint64)
        for done in range(2):
            tot += O.mc_sweep(mp, done, domain, None, spin)
        assert mc.sweep(2) == int(tot[1])
        assert np.array_equal(mc.crystals(), spin)
        mc.close()
