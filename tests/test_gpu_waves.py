"""The kernels with one warp per neighbour column are compiled for two to five blocks an
SM and chosen by the grid: every choice, at the slot counts where it changes, against the
oracle (FP64 steps, bit for bit) and the kernels with one thread per slot (adjoint)."""
import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, configs
from boltzmannmfx_gb300.abi import BMXG_FP64

pytestmark = pytest.mark.gpu

OUT = ("x", "y", "z", "velx", "vely", "velz")
WAVE = 152 * 32  # slots of one block an SM
EDGES = [2 * WAVE, 2 * WAVE + 1, 3 * WAVE, 3 * WAVE + 1, 4 * WAVE, 4 * WAVE + 1, 5 * WAVE, 5 * WAVE + 1, 6 * WAVE + 1]


def colony(n):
    side = 0.192
    P = configs.sphere_colony(n, side, side, np.random.default_rng(n))
    rng = np.random.default_rng(n + 1)
    for k, c in (("x", 0.0110), ("y", 0.0110), ("z", 0.0450)):  # a crowd inside one bin
        P[k][:40] = c + rng.uniform(-4.0e-4, 4.0e-4, 40)
    return configs.deck_params(), configs.box_geometry(side, side), P


@pytest.mark.parametrize("n", EDGES)
def test_fp64_steps_bit_exact(gpu_lib, oracle_lib, n):
    prm, g, P = colony(n)
    ctx = Context(prm, [g])
    ctx.set_state(P)
    ctx.step(0.25, 2, BMXG_FP64)
    Q, R = P.copy(), P.copy()
    ctx.get_state(Q)
    ctx.close()
    oracle_lib.evolve(prm, [g], [0, n], R, 0.25, 2)
    for k in OUT:
        assert np.array_equal(Q[k], R[k]), k


@pytest.mark.parametrize("n", EDGES)
def test_adjoint_equals_one_thread_per_slot(gpu_lib, n):
    prm, g, P = colony(n)
    rng = np.random.default_rng(n)
    adh, grad = rng.uniform(0.0, 1.0e-3, n), rng.normal(0.0, 1.0, (3, n))
    got = []
    for grid in (0, 4096):
        ctx = Context(prm, [g])
        if grid:
            ctx.set_shapes(sphere_grid=[grid, 0], sphere_block=[64, 64])
        ctx.set_state(P)
        ctx.set_ext(0.05, 1.0e-2, adh)
        ctx.forward(0.25, 3, 2)
        Q = P.copy()
        ctx.get_state(Q)
        got.append([Q[k] for k in OUT[:3]] + list(ctx.backward(grad)))
        ctx.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
