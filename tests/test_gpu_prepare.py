"""bmxg_prepare where FP64 steps take the neighbour list instantiates the graphs of the
steps without it as well: calls of one to nine steps after it, on the list and after a
load off it, give the results of an unprepared context."""
import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, configs
from boltzmannmfx_gb300.abi import BMXG_FP64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reload", [False, True])
def test_calls_after_prepare(gpu_lib, reload):
    n, side = 30_000, 0.256
    g, P = configs.box_geometry(side, side), configs.sphere_colony(n, side, side, np.random.default_rng(71))
    got = []
    for prepare in (True, False):
        ctx = Context(configs.deck_params(), [g])
        ctx.set_state(P)
        ctx.step(0.25, 160, BMXG_FP64)
        assert ctx.stats()["n_rebins"] < 160
        ctx.set_state(P)
        if prepare:
            ctx.prepare(0.25, BMXG_FP64)
        if reload:
            ctx.set_state(P)
        out = []
        for steps in (1, 2, 1, 9):
            ctx.step(0.25, steps, BMXG_FP64)
            Q = P.copy()
            ctx.get_state(Q)
            out += [Q[k] for k in ("x", "y", "z", "velx", "vely", "velz")]
        got.append(out)
        ctx.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
