"""The FP64 step with one thread per slot (k_sphere64) over the column-sorted
copies, and the rule that chooses it, against the oracle, bit for bit: slot counts
around the rule's limit and a block, closed and periodic faces, columns taller than a
search's threshold, and slots around and beyond the staged candidates."""
import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, configs
from boltzmannmfx_gb300.abi import BMXG_FP64, Geometry

pytestmark = pytest.mark.gpu

OUT = ("x", "y", "z", "velx", "vely", "velz")


@pytest.mark.parametrize("n, side, crowd, per, pinned", [
    (32768, 0.256, 12, 1, False), (32769, 0.256, 13, 1, False), (32831, 0.256, 14, 0, False),
    (40000, 0.128, 0, 1, False), (33000, 0.256, 60, 1, False), (1, 0.006, 0, 1, True), (63, 0.006, 0, 1, True),
    (65, 0.016, 40, 0, True), (3000, 0.032, 0, 1, True)])
def test_steps_bit_exact(gpu_lib, oracle_lib, n, side, crowd, per, pinned):
    prm = configs.deck_params()
    m = int(round(side / configs.BIN))
    g = Geometry.make((0.0, 0.0, 0.0), (side, side, 0.064), (m, m, 32), (per, per, 0))
    P = configs.sphere_colony(n, side, side, np.random.default_rng(n))
    rng = np.random.default_rng(n + 1)
    for k, c in (("x", 0.0110), ("y", 0.0110), ("z", 0.0450)):  # a crowd inside one bin
        P[k][:crowd] = c + rng.uniform(-4.0e-4, 4.0e-4, crowd)
    ctx = Context(prm, [g])
    if pinned:
        ctx.set_shapes(sphere_grid=[7, 0], sphere_block=[64, 64])
    ctx.set_state(P)
    ctx.step(0.25, 2, BMXG_FP64)
    Q = P.copy()
    ctx.get_state(Q)
    ctx.close()
    R = P.copy()
    oracle_lib.evolve(prm, [g], [0, n], R, 0.25, 2)
    for k in OUT:
        assert np.array_equal(Q[k], R[k]), k
