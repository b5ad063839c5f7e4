"""The tile step on both sides of its block size rule, with crowded cells (more
candidates than a column's staging holds), a tile of one cell across, and
particles at the closed z faces: bit for bit the whole-domain step."""
import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, configs

from test_gpu_tile import OUT, tile_inputs, whole_domain_step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, side, lo, hi, crowd", [
    (40, 0.016, (0, 0, 0), (7, 7, 31), 0),
    (300, 0.016, (3, 0, 0), (3, 7, 31), 0),
    (2000, 0.064, (0, 8, 20), (15, 31, 24), 60),
    (70_000, 0.256, (0, 0, 0), (127, 127, 31), 50),
    (90_000, 0.256, (1, 0, 0), (120, 127, 31), 0)])
def test_tile_equals_whole_domain(gpu_lib, n, side, lo, hi, crowd):
    rng = np.random.default_rng(n)
    prm, g = configs.deck_params(), configs.box_geometry(side, side)
    P = configs.sphere_colony(n, side, side, rng)
    P["x"][:crowd] = (lo[0] + 0.5) * configs.BIN + rng.uniform(-3.0e-4, 3.0e-4, crowd)
    P["y"][:crowd] = (lo[1] + 0.5) * configs.BIN + rng.uniform(-3.0e-4, 3.0e-4, crowd)
    P["z"][:crowd] = 0.0451 + rng.uniform(-3.0e-4, 3.0e-4, crowd)
    P["z"][crowd:crowd + 3] = (-0.0005, 0.0639, 0.0642)     # below, at and above the closed faces
    ref = whole_domain_step(prm, g, P, 0.25)
    idx, R, G = tile_inputs(g, P, lo, hi)
    assert len(idx) > 0
    ctx = Context(prm, [g])
    ctx.step_tile(lo, hi, R, G, 0.25)
    ctx.close()
    for k in OUT:
        assert np.array_equal(R[k], ref[k][idx]), k
