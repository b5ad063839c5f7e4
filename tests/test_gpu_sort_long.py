"""The column sort where columns are long (tall domains): the runs of 128 keys that
are sorted first, at the edges of their length and of the rule's, in the cluster
sort and in the separate kernels (whole domains and tiles).  Neighbour lists and
FP64 steps equal the oracle's, which needs every column's order."""
import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, configs
from boltzmannmfx_gb300.abi import BMXG_FP64, Geometry
from oracle import oracle as O

from common import same_pairs
from test_gpu_tile import OUT, tile_inputs, whole_domain_step

pytestmark = pytest.mark.gpu

PRM = configs.deck_params()


def tall(n, mx, my, nz, seed, per=0):
    lx, ly, lz = mx * configs.BIN, my * configs.BIN, nz * configs.BIN
    g = Geometry.make((0.0, 0.0, 0.0), (lx, ly, lz), (mx, my, nz), (per, per, 0))
    P = configs.sphere_colony(n, lx, ly, np.random.default_rng(seed), z_band=(0.0, lz))
    return g, P


# one column of a length around the rule's and the runs' edges; several columns, one of them
# long; the cluster's last size and the separate kernels
@pytest.mark.parametrize("n, mx, my, nz", [
    (127, 1, 1, 40), (160, 1, 1, 50), (161, 1, 1, 50), (255, 1, 1, 60), (256, 1, 1, 60), (257, 1, 1, 60),
    (1500, 1, 1, 300), (5000, 3, 3, 160), (20_000, 2, 5, 900), (65_536, 4, 8, 900), (65_537, 4, 8, 900),
    (70_001, 3, 3, 3000)])
def test_long_columns(gpu_lib, n, mx, my, nz):
    g, P = tall(n, mx, my, nz, n, 1 if mx > 2 and my > 2 else 0)
    if mx * my == 9:  # an uneven load: a third of the slots in one column
        P["x"][::3] = np.random.default_rng(1).uniform(0.0, configs.BIN, P["x"][::3].size)
        P["y"][::3] = np.random.default_rng(2).uniform(0.0, configs.BIN, P["y"][::3].size)
    ctx = Context(PRM, [g])
    ctx.set_state(P)
    if n <= 20_000:
        assert same_pairs(ctx.pairs(), O.pairs(PRM, g, P))
    ctx.step(0.25, 2, BMXG_FP64)
    Q, R = P.copy(), P.copy()
    ctx.get_state(Q)
    ctx.close()
    O.evolve(PRM, [g], [0, n], R, 0.25, 2)
    for k in ("x", "y", "z", "velx", "vely", "velz"):
        assert np.array_equal(Q[k], R[k]), k


@pytest.mark.parametrize("n, m, nz", [(9000, 6, 300), (120_000, 6, 4000)])
def test_tile_of_long_columns(gpu_lib, n, m, nz):
    g, P = tall(n, m, m, nz, n, 1)
    lo, hi = (0, 1, 0), (3, 4, nz - 1)
    ref = whole_domain_step(PRM, g, P, 0.25)
    idx, R, G = tile_inputs(g, P, lo, hi)
    ctx = Context(PRM, [g])
    ctx.step_tile(lo, hi, R, G, 0.25)
    ctx.close()
    for k in OUT:
        assert np.array_equal(R[k], ref[k][idx]), k


@pytest.mark.parametrize("n, crowd", [(3000, 161), (3000, 1500), (70_000, 900)])
def test_one_long_column_among_many(gpu_lib, n, crowd):
    """A column that the average does not show: found by the load's sort, and gone with
    the next load; a column that grows long during the steps likewise."""
    m, nz = 64, 400
    g, P = tall(n, m, m, nz, n, 1)
    L = P.copy()
    rng = np.random.default_rng(n + 1)
    L["x"][:crowd] = 0.0210 + rng.uniform(-9.0e-4, 9.0e-4, crowd)
    L["y"][:crowd] = 0.0210 + rng.uniform(-9.0e-4, 9.0e-4, crowd)
    ctx = Context(PRM, [g])
    for S in (L, P, L):
        ctx.set_state(S)
        for steps in (1, 9):
            ctx.step(0.25, steps, BMXG_FP64)
        Q, R = S.copy(), S.copy()
        ctx.get_state(Q)
        O.evolve(PRM, [g], [0, n], R, 0.25, 10)
        for k in ("x", "y", "z", "velx", "vely", "velz"):
            assert np.array_equal(Q[k], R[k]), k
        if n <= 20_000:
            assert same_pairs(ctx.pairs(), O.pairs(PRM, g, Q))
    ctx.close()


@pytest.mark.parametrize("n, mx, my", [(700, 256, 256), (700, 257, 256), (40_000, 256, 256), (40_000, 255, 258)])
def test_column_counts_around_the_cluster_sorts(gpu_lib, n, mx, my):
    """65 536 columns and a few more."""
    g, P = tall(n, mx, my, 32, n + mx, 1)
    ctx = Context(PRM, [g])
    ctx.set_state(P)
    if n <= 20_000:
        assert same_pairs(ctx.pairs(), O.pairs(PRM, g, P))
    ctx.step(0.25, 3, BMXG_FP64)
    Q, R = P.copy(), P.copy()
    ctx.get_state(Q)
    ctx.close()
    O.evolve(PRM, [g], [0, n], R, 0.25, 3)
    for k in ("x", "y", "z", "velx", "vely", "velz"):
        assert np.array_equal(Q[k], R[k]), k
