"""Sweeps of a listed domain (mc.domain = basalt) on the byte copy of its orientations, against the CPU
oracle, bit for bit: one block and many, one entry per thread and colour and several, every
neighbourhood and boundary, rows of any remainder, the largest Q of the byte form, and the calls that
take the 32-bit form instead (Q > 256, orientations set from outside, rows below six cells)."""
import numpy as np
import pytest

from oracle import oracle as O
from volcano_ca_mc_b200 import capi

pytestmark = pytest.mark.gpu

CASES = [
    # nb, bc, dims, share of the cells, Q, kT, mobility
    ("moore", "periodic", (6, 7, 8), 0.7, 20, 0.7, False),
    ("moore", "absorbing", (17, 13, 11), 0.5, 256, 0.6, True),
    ("pentagonal", "periodic", (23, 15, 10), 0.6, 256, 0.5, True),
    ("von_neumann", "periodic", (9, 10, 7), 0.5, 2, 0.5, False),
    ("von_neumann", "absorbing", (30, 1, 41), 0.4, 33, 0.0, True),
    ("hexagonal", "periodic", (37, 1, 52), 0.5, 64, 0.6, True),
    ("pentagonal", "absorbing", (50, 1, 29), 0.9, 129, 0.6, False),
    ("moore", "periodic", (64, 50, 40), 0.3, 128, 0.6, True),       # many blocks
    ("moore", "periodic", (65, 2, 33), 0.8, 100, 0.4, False),       # a 2-cell wrapped axis, a third colour class
    ("von_neumann", "absorbing", (100, 80, 60), 0.8, 77, 0.5, True),  # two entries per thread and colour
    ("moore", "absorbing", (17, 13, 11), 0.5, 300, 0.6, True),      # the 32-bit form
    ("moore", "periodic", (5, 13, 11), 0.5, 50, 0.6, False),        # the 32-bit form
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}-{c[1]}-{'x'.join(map(str, c[2]))}-Q{c[4]}")
def test_list_sweeps_match_oracle(case):
    nb, bc, (nx, ny, nz), share, Q, kT, use_mob = case
    seed = 11 + nx + 3 * ny
    n = nx * ny * nz
    rng = np.random.default_rng(seed)
    domain = (rng.random(n) < share).astype(np.uint8)
    mob = (rng.uniform(0.2, 1.0, n) * domain).astype(np.float32) if use_mob else None
    mp = O.mc_params(nx, ny, nz, nb, bc, False, seed, Q, 1.0, kT)
    spin = O.mc_init(mp, domain)
    mc = capi.PottsMC(capi.McParams(nx, ny, nz, neighborhood=nb, boundary=bc, seed=seed, Q=Q, kT=kT))
    mc.set_domain(domain)
    if use_mob:
        mc.set_mobility(mob)
    mc.initialize()
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
    # orientations from outside, then on
    spin = np.where(domain, rng.integers(1, Q + 1, n), 0).astype(np.int32)
    mc.set_spins(spin)
    for _ in range(2):
        O.mc_sweep(mp, done, domain, mob, spin)
        done += 1
    mc.sweep(2)
    assert np.array_equal(mc.crystals(), spin)
    mc.close()
