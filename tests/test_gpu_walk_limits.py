"""Both sides of the slot counts up to which a warp takes a neighbour column: FP64 steps
against the oracle, the adjoint against the kernels with one thread per slot (pinned
launch shapes), bit for bit."""
import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, configs
from boltzmannmfx_gb300.abi import BMXG_FP64

pytestmark = pytest.mark.gpu

OUT = ("x", "y", "z", "velx", "vely", "velz")
PRM = configs.deck_params()


@pytest.mark.parametrize("n", [49152, 49153])
def test_steps(gpu_lib, oracle_lib, n):
    side = 0.256
    g, P = configs.box_geometry(side, side), configs.sphere_colony(n, side, side, np.random.default_rng(n))
    ctx = Context(PRM, [g])
    ctx.set_state(P)
    ctx.step(0.25, 2, BMXG_FP64)
    Q, R = P.copy(), P.copy()
    ctx.get_state(Q)
    ctx.close()
    oracle_lib.evolve(PRM, [g], [0, n], R, 0.25, 2)
    for k in OUT:
        assert np.array_equal(Q[k], R[k]), k


@pytest.mark.parametrize("n", [65536, 65537, 114688, 114689])
def test_adjoint(gpu_lib, n):
    side = 0.384
    g, P = configs.box_geometry(side, side), configs.sphere_colony(n, side, side, np.random.default_rng(n))
    rng = np.random.default_rng(n + 1)
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
