"""Calls of few list steps (each step counts itself) and of more (set before the
call), mixed, give the trajectory and the counters of one long call."""
import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, configs
from boltzmannmfx_gb300.abi import BMXG_FP32F, BMXG_FP64

pytestmark = pytest.mark.gpu

OUT = ("x", "y", "z", "velx", "vely", "velz")


@pytest.mark.parametrize("n, side, prec", [(3000, 0.128, BMXG_FP32F), (400100, 0.9, BMXG_FP32F), (16800, 0.184, BMXG_FP64)])
@pytest.mark.parametrize("calls", [(1, 1, 2, 3, 4, 5, 9, 1, 2), (8, 1, 16, 2, 1)])
@pytest.mark.parametrize("prepared", [False, True])
def test_split_calls_equal_one_call(gpu_lib, n, side, prec, calls, prepared):
    prm, g = configs.deck_params(), configs.box_geometry(side, side)
    P = configs.sphere_colony(n, side, side, np.random.default_rng(n))
    got = []
    for parts in (calls, (sum(calls),)):
        ctx = Context(prm, [g])
        ctx.set_state(P)
        ctx.step(0.25, 160 if prec == BMXG_FP64 else 8, prec)
        if prepared:
            ctx.prepare(0.25, prec)
        r0 = ctx.stats()["n_rebins"]
        for k in parts:
            ctx.step(0.25, k, prec)
        Q = P.copy()
        ctx.get_state(Q)
        s = ctx.stats()
        assert s["n_rebins"] - r0 < sum(calls)
        got.append([Q[k] for k in OUT] + [s["n_out_of_domain"], s["n_edge_ghost"], s["n_rebins"]])
        ctx.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
