"""Grain statistics on the device (labelGrains, engine/src/mc/Grains.cpp:33-150; the classes of
McStage, engine/src/app/McStage.cpp:38-66) against connected components on the host: spaces with fewer
and with more cells than the launch has threads, one grain and many, partial domains, both
connectivities."""
import numpy as np
import pytest
from scipy.sparse import coo_matrix
from scipy.sparse.csgraph import connected_components

from volcano_ca_mc_b200 import capi

pytestmark = pytest.mark.gpu


def _host(spins, dims, moore, periodic, mob, threshold):
    nx, ny, nz = dims
    n = spins.size
    s = spins.reshape(nz, ny, nx)
    idx = np.arange(n).reshape(nz, ny, nx)
    rows, cols = [], []
    for dz in (0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                if not (dz > 0 or (dz == 0 and (dy > 0 or (dy == 0 and dx > 0)))):
                    continue
                if (nx == 1 and dx) or (ny == 1 and dy) or (nz == 1 and dz) or (not moore and abs(dx) + abs(dy) + abs(dz) != 1):
                    continue
                q, t = np.roll(idx, (-dz, -dy, -dx), (0, 1, 2)), np.roll(s, (-dz, -dy, -dx), (0, 1, 2))
                ok = (s == t) & (s > 0)
                if not periodic:
                    for axis, d, size in ((2, dx, nx), (1, dy, ny), (0, dz, nz)):
                        if d:
                            edge = np.zeros_like(ok)
                            edge[tuple(slice(None) if a != axis else (size - 1 if d > 0 else 0) for a in range(3))] = True
                            ok &= ~edge
                rows.append(idx[ok])
                cols.append(q[ok])
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    _, label = connected_components(coo_matrix((np.ones(len(rows), np.int8), (rows, cols)), shape=(n, n)), directed=False)
    on = spins > 0
    label = label[on]
    high = (mob[on].astype(np.float64) >= threshold) if mob is not None else np.zeros(on.sum(), bool)
    _, inv = np.unique(label, return_inverse=True)
    size, hi = np.bincount(inv), np.bincount(inv, weights=high).astype(int)
    up = 2 * hi >= size
    most = lambda v: int(v.max()) if len(v) else 0
    return (len(size), int(on.sum()), most(size), int(high.sum()), int(up.sum()), int(size[up].sum()), most(size[up]),
            int((~up).sum()), int(size[~up].sum()), most(size[~up]))


@pytest.mark.parametrize("case", [((70, 60, 50), "moore", "periodic", 2, 1.0, True), ((70, 60, 50), "von_neumann", "absorbing", 3, 1.0, False),
                                  ((64, 50, 60), "moore", "absorbing", 40, 0.6, True), ((90, 80, 1), "moore", "periodic", 1, 1.0, False),
                                  ((16, 16, 1), "von_neumann", "periodic", 2, 0.5, True), ((400, 1, 500), "von_neumann", "periodic", 4, 0.9, True)],
                         ids=lambda c: f"{'x'.join(map(str, c[0]))}-{c[1]}-{c[2]}-{c[3]}")
def test_grain_statistics_match_connected_components(case):
    dims, nb, bc, kinds, share, use_mob = case
    rng = np.random.default_rng(sum(dims))
    n = int(np.prod(dims))
    domain = (rng.random(n) < share).astype(np.uint8)
    spins = np.where(domain, rng.integers(1, kinds + 1, n), 0).astype(np.int32)
    mob = rng.random(n).astype(np.float32) * domain if use_mob else None
    mc = capi.PottsMC(capi.McParams(*dims, neighborhood=nb, boundary=bc, domain_full=True, seed=1, Q=64))
    mc.set_domain(domain)
    if use_mob:
        mc.set_mobility(mob)
    mc.initialize()
    mc.set_spins(spins)
    for _ in range(2):  # a second call on the same buffers
        g = mc.grains(moore=nb == "moore", threshold=0.5)
        got = (g.grains, g.cells, g.largest, g.high_cells, g.high_grains, g.high_grain_cells, g.high_largest, g.low_grains,
               g.low_grain_cells, g.low_largest)
        assert got == _host(spins, dims, nb == "moore", bc == "periodic", mob, 0.5)
    mc.close()


@pytest.mark.parametrize("listed", [False, True], ids=["whole", "partial"])
@pytest.mark.parametrize("nb", ["moore", "von_neumann"])
@pytest.mark.parametrize("dims", [(33, 6, 5), (64, 5, 4), (2, 3, 5), (3, 2, 2), (1, 7, 9), (100, 2, 1)], ids=lambda d: "x".join(map(str, d)))
def test_grains_of_whole_rows(dims, nb, listed):
    """Runs as long as their row, rings on a periodic axis, pairs of rows that only their ends join, axes of
    one to three cells."""
    nx, ny, nz = dims
    rng = np.random.default_rng(nx + 7 * ny)
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    for periodic in (True, False):
        for k, spins in enumerate((1 + y // 2 % 2 + 2 * (z % 2), 1 + (x + y) // 3 % 2, np.where(x == nx - 1, 1, 2 + (y + z) % 2),
                                   rng.integers(1, 3, (nz, ny, nx)))):
            spins = spins.astype(np.int32).reshape(-1)
            domain = np.ones(spins.size, np.uint8)
            if listed:
                domain[rng.integers(0, spins.size, max(1, spins.size // 9))] = 0
                spins = spins * domain
            mc = capi.PottsMC(capi.McParams(*dims, neighborhood=nb, boundary="periodic" if periodic else "absorbing", domain_full=True,
                                            seed=1, Q=64))
            mc.set_domain(domain)
            mc.initialize()
            mc.set_spins(spins)
            g = mc.grains(moore=nb == "moore", threshold=0.5)
            got = (g.grains, g.cells, g.largest, g.high_cells, g.high_grains, g.high_grain_cells, g.high_largest, g.low_grains,
                   g.low_grain_cells, g.low_largest)
            assert got == _host(spins, dims, nb == "moore", periodic, None, 0.5), (periodic, k)
            mc.close()
