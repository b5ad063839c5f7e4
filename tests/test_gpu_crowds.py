"""FP64 sphere steps and the adjoint where slots have as many candidates as the kernels
stage and one more (12 in a neighbour column with a warp per column, 24 in all with a
thread per slot), the crowd inside a bin, across bins and around a periodic corner,
whose images are staged with the shift: bit for bit the oracle's steps, and the
adjoint of the kernels with one thread per slot."""
import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, configs
from boltzmannmfx_gb300.abi import BMXG_FP64

pytestmark = pytest.mark.gpu

OUT = ("x", "y", "z", "velx", "vely", "velz")
PRM = configs.deck_params()


def crowded(n, side, crowd, at, seed):
    P = configs.sphere_colony(n, side, side, np.random.default_rng(seed))
    rng = np.random.default_rng(seed + 1)
    for k, c in zip(("x", "y"), at):
        P[k][:crowd] = (c + rng.uniform(-2.5e-4, 2.5e-4, crowd)) % side
    P["z"][:crowd] = 0.0450 + rng.uniform(-2.5e-4, 2.5e-4, crowd)
    return P


@pytest.mark.parametrize("n, side", [(200, 0.064), (33_000, 0.256)])
@pytest.mark.parametrize("crowd", [12, 13, 14, 24, 25, 26, 48, 60])
@pytest.mark.parametrize("at", [(0.011, 0.011), (0.012, 0.012), (0.0, 0.0)])
def test_steps_bit_exact(gpu_lib, oracle_lib, n, side, crowd, at):
    g, P = configs.box_geometry(side, side), crowded(n, side, crowd, at, crowd)
    ctx = Context(PRM, [g])
    ctx.set_state(P)
    ctx.step(0.25, 2, BMXG_FP64)
    Q, R = P.copy(), P.copy()
    ctx.get_state(Q)
    edge = ctx.stats()["n_edge_ghost"]
    ctx.close()
    oracle_lib.evolve(PRM, [g], [0, n], R, 0.25, 2)
    assert edge == 0
    for k in OUT:
        assert np.array_equal(Q[k], R[k]), k


@pytest.mark.parametrize("crowd, at", [(12, (0.012, 0.012)), (13, (0.011, 0.011)), (26, (0.0, 0.0)),
                                       (52, (0.0, 0.011))])
def test_adjoint_equals_one_thread_per_slot(gpu_lib, crowd, at):
    n, side = 3000, 0.064
    g, P = configs.box_geometry(side, side), crowded(n, side, crowd, at, crowd)
    rng = np.random.default_rng(crowd)
    adh, grad = rng.uniform(0.0, 1.0e-3, n), rng.normal(0.0, 1.0, (3, n))
    got = []
    for grid in (0, 4096):
        ctx = Context(PRM, [g])
        if grid:
            ctx.set_shapes(sphere_grid=[grid, 0], sphere_block=[64, 64])
        ctx.set_state(P)
        ctx.set_ext(0.05, 1.0e-2, adh)
        ctx.forward(0.25, 3, 2)
        Q = P.copy()
        ctx.get_state(Q)
        got.append([Q[k] for k in OUT] + list(ctx.backward(grad)))
        ctx.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
