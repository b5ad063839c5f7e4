"""The column sort in one thread-block cluster (k_sort_cluster) and its separate
kernels, at the edges of its sizes: one slot, a block's and the cluster's
threads and items per thread and one more, few and many columns.  After a load
and after a step the neighbour list equals the oracle's entry for entry, which
needs every column's offsets and order; the step's counters are the last
step's."""
import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, configs
from boltzmannmfx_gb300.abi import BMXG_FP64
from oracle import oracle as O

from common import same_pairs

pytestmark = pytest.mark.gpu


def colony(n, side, seed):
    rng = np.random.default_rng(seed)
    return configs.deck_params(), configs.box_geometry(side, side), configs.sphere_colony(n, side, side, rng)


@pytest.mark.parametrize("n, side", [(1, 0.006), (2, 0.064), (1023, 0.006), (1024, 0.128), (1025, 0.032),
                                     (16385, 0.128), (65536, 0.256), (65537, 0.256), (3000, 1.024), (3000, 1.1)])
def test_sorted_columns_give_the_oracles_list(gpu_lib, n, side):
    prm, g, P = colony(n, side, n)
    ctx = Context(prm, [g])
    ctx.set_state(P)
    if n <= 20000:
        assert same_pairs(ctx.pairs(), O.pairs(prm, g, P))
    ctx.step(0.25, 3, BMXG_FP64)
    Q = P.copy()
    ctx.get_state(Q)
    R = P.copy()
    O.evolve(prm, [g], [0, n], R, 0.25, 3)
    for k in ("x", "y", "z", "velx", "vely", "velz"):
        assert np.array_equal(Q[k], R[k]), k
    if n <= 20000:
        assert same_pairs(ctx.pairs(), O.pairs(prm, g, Q))
    ctx.close()


@pytest.mark.parametrize("n", [40, 70_000])
def test_counters_are_the_last_steps(gpu_lib, n):
    """Slots outside the closed z range are counted once per step, not summed
    over the steps of a call or over calls."""
    prm, g, P = colony(n, 0.256, 3)
    P["z"][:5] = 0.0641 + 1.0e-4 * np.arange(5)
    ctx = Context(prm, [g])
    ctx.set_state(P)
    for steps in (1, 9, 2):
        ctx.step(0.25, steps, BMXG_FP64)
        assert ctx.stats()["n_out_of_domain"] == 5
    ctx.close()
