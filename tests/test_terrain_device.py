"""Spill levels and ROCK columns of vca_ca_apply_terrain against the oracle's priority flood
(TerrainGenerator::fillDepressions, engine/src/terrain/TerrainGenerator.cpp:86-161): maps on both sides
of the line between the host's and the device's flood, whole and partial tiles, wrapped and open axes,
noise, cones, basins inside basins and long winding valleys."""
import numpy as np
import pytest

from oracle import oracle as O
from volcano_ca_mc_b200 import capi

pytestmark = pytest.mark.gpu


def _map(kind, nx, ny, seed):
    rng = np.random.default_rng(seed)
    x, y = np.arange(nx)[None, :], np.arange(ny)[:, None]
    if kind == "noise":
        h = rng.integers(0, 40, size=(ny, nx))
    elif kind == "basins":  # rings of ridges of rising height with noise, a breach in each
        r = np.sqrt((x - nx / 2) ** 2 + (y - ny / 2) ** 2)
        h = np.where((r.astype(int) // 9) % 2 == 0, 4, 30 - (r / 12).astype(int) % 20) + rng.integers(0, 4, size=(ny, nx))
        h[ny // 2, :] = np.minimum(h[ny // 2, :], 9)
    elif kind == "winding":  # a serpentine valley between high walls
        h = np.full((ny, nx), 45)
        for j in range(1, ny - 1, 4):
            h[j, 1:nx - 1] = 3 + rng.integers(0, 3, size=nx - 2)
            h[min(j + 1, ny - 1):min(j + 4, ny - 1), (nx - 2) if (j // 4) % 2 == 0 else 1] = 5
        h[min(1, ny - 1), 0] = 2
    else:
        h = 40 * np.exp(-((x - nx / 3) ** 2 + (y - ny / 2) ** 2) / (2 * (nx / 5) ** 2)) + rng.uniform(0, 3, size=(ny, nx))
    return np.clip(h, 0, 60).astype(np.int32).reshape(-1)


@pytest.mark.parametrize("kind", ["noise", "basins", "winding", "cone"])
@pytest.mark.parametrize("size", [(90, 91), (96, 96), (128, 64), (257, 129), (33, 300), (9000, 1), (300, 290), (64, 40),
                                  (60, 42)],
                         ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("boundary", ["absorbing", "periodic"])
def test_spill_levels_match_oracle(kind, size, boundary):
    nx, ny = size
    nz = 20  # some columns are higher than the space
    h = _map(kind, nx, ny, nx + ny)
    per = boundary == "periodic"
    ca = capi.LavaCA(capi.CaParams(nx, ny, nz, neighborhood="moore", boundary=boundary, seed=1, max_steps=5))
    ca.apply_terrain(h)
    assert np.array_equal(ca.spill(), O.fill_depressions(h, nx, ny, per and nx > 1, per and ny > 1))
    ca.place_seeds([])
    types = ca.download()[0].reshape(nz, ny, nx)
    want = np.arange(nz)[:, None, None] < h.reshape(ny, nx)[None]
    assert np.array_equal(types, want.astype(np.uint8))
    ca.close()


def test_negative_height_keeps_the_terrain():
    nx, ny, nz = 128, 100, 8
    h = _map("noise", nx, ny, 3) % 8
    ca = capi.LavaCA(capi.CaParams(nx, ny, nz, seed=1, max_steps=5))
    ca.apply_terrain(h)
    spill = ca.spill()
    bad = h.copy()
    bad[77] = -1
    with pytest.raises(capi.VcaError, match="negative height"):
        ca.apply_terrain(bad)
    assert np.array_equal(ca.spill(), spill)
    ca.close()
