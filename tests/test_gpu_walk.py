"""The FP64 kernels with one warp per neighbour column (k_sphere64w, k_dfwdw,
k_dadjw) against the oracle, bit for bit, and against the kernels with one
thread per slot: sizes around a block's slots and around the launch rule's
limits, closed and periodic faces, and columns more crowded than the staging
holds (those slots walk serially)."""
import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, configs
from boltzmannmfx_gb300.abi import BMXG_FP64, Geometry
from oracle import oracle as O

pytestmark = pytest.mark.gpu

OUT = ("x", "y", "z", "velx", "vely", "velz")


def colony(n, side, crowd, seed):
    P = configs.sphere_colony(n, side, side, np.random.default_rng(seed))
    rng = np.random.default_rng(seed + 1)
    for k, c in (("x", 0.0110), ("y", 0.0110), ("z", 0.0450)):  # a crowd inside one bin
        P[k][:crowd] = c + rng.uniform(-4.0e-4, 4.0e-4, crowd)
    return P


@pytest.mark.parametrize("n, side, crowd, per", [
    (1, 0.006, 0, 1), (31, 0.006, 0, 1), (33, 0.016, 0, 0), (64, 0.032, 60, 1), (129, 0.032, 9, 1),
    (1000, 0.032, 8, 0), (65536, 0.324, 40, 1), (65537, 0.324, 40, 1), (65665, 0.324, 0, 0)])
def test_fp64_steps_bit_exact(gpu_lib, n, side, crowd, per):
    prm = configs.deck_params()
    m = int(round(side / configs.BIN))
    g = Geometry.make((0.0, 0.0, 0.0), (side, side, 0.064), (m, m, 32), (per, per, 0))
    P = colony(n, side, crowd, n)
    ctx = Context(prm, [g])
    ctx.set_state(P)
    ctx.step(0.25, 2, BMXG_FP64)
    Q = P.copy()
    ctx.get_state(Q)
    ctx.close()
    R = P.copy()
    O.evolve(prm, [g], [0, n], R, 0.25, 2)
    for k in OUT:
        assert np.array_equal(Q[k], R[k]), k


@pytest.mark.parametrize("n, crowd", [(1, 0), (33, 20), (2000, 50), (4001, 0)])
def test_adjoint_equals_one_thread_per_slot(gpu_lib, n, crowd):
    """Pinned launch shapes select the kernels with one thread per slot."""
    prm, g = configs.deck_params(), configs.box_geometry(0.064, 0.064)
    P = colony(n, 0.064, crowd, n)
    rng = np.random.default_rng(n)
    adh, grad = rng.uniform(0.0, 1.0e-3, n), rng.normal(0.0, 1.0, (3, n))
    got = []
    for grid in (0, 4096):
        ctx = Context(prm, [g])
        if grid:
            ctx.set_shapes(sphere_grid=[grid, 0], sphere_block=[64, 64])
        ctx.set_state(P)
        ctx.set_ext(0.05, 1.0e-2, adh)
        ctx.forward(0.25, 5, 2)
        Q = P.copy()
        ctx.get_state(Q)
        got.append([Q[k] for k in OUT] + list(ctx.backward(grad)))
        ctx.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
