"""FP64 steps whose lists do not last (a reader of the bins, the other form or a load
after every step or few, steps so long that every one needs a build) settle on the
per-step path: after a few rounds a round enqueues the kernels that it enqueues with
the list off, and the results are the same throughout."""
import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, configs
from boltzmannmfx_gb300.abi import BMXG_FP32F, BMXG_FP64

pytestmark = pytest.mark.gpu

OUT = ("x", "y", "z", "velx", "vely", "velz")


def rounds(ctx, kind, P):
    if kind == "export":
        ctx.step(0.25, 1, BMXG_FP64)
        return ctx.pairs()
    if kind == "loads":
        ctx.set_state(P)
        for _ in range(7):
            ctx.step(0.25, 1, BMXG_FP64)
    elif kind == "fast":
        ctx.set_state(P)
        ctx.step(8.0, 12, BMXG_FP64)
    return None


@pytest.mark.parametrize("kind", ["export", "loads", "fast"])
def test_short_lists(gpu_lib, kind):
    n, side = 17000, 0.184
    prm, g = configs.deck_params(), configs.box_geometry(side, side)
    P = configs.sphere_colony(n, side, side, np.random.default_rng(31))
    A, B = Context(prm, [g]), Context(prm, [g])
    B.set_list_mode(0)
    for c in (A, B):
        c.set_state(P)
        c.step(0.25, 160, BMXG_FP64)  # (the list's buffers are paid for)
    assert A.stats()["n_rebins"] < 160
    for r in range(10):
        took = []
        for c in (A, B):
            l0 = c.stats()["n_kernel_launches"]
            c.got = rounds(c, kind, P)
            took.append(c.stats()["n_kernel_launches"] - l0)
        QA, QB = P.copy(), P.copy()
        A.get_state(QA)
        B.get_state(QB)
        for k in OUT:
            assert np.array_equal(QA[k], QB[k]), k
        if kind == "export":
            assert all(np.array_equal(x, y) for x, y in zip(A.got, B.got))
    assert took[0] == took[1]
    # and back to the list where the steps are many
    A.set_state(P)
    r0 = A.stats()["n_rebins"]
    A.step(0.25, 80, BMXG_FP64)
    assert A.stats()["n_rebins"] - r0 < 40
    A.close()
    B.close()


def test_one_step_between_steps_of_the_other_form(gpu_lib):
    n, side = 17000, 0.184
    prm, g = configs.deck_params(), configs.box_geometry(side, side)
    P = configs.sphere_colony(n, side, side, np.random.default_rng(37))
    A, B = Context(prm, [g]), Context(prm, [g])
    for c in (A, B):
        c.set_state(P)
        c.step(0.25, 160, BMXG_FP64)
    for r in range(8):
        A.step(0.25, 4, BMXG_FP32F)
        l0 = A.stats()["n_kernel_launches"]
        A.step(0.25, 1, BMXG_FP64)
        took = A.stats()["n_kernel_launches"] - l0
    assert took <= 5  # the positions, a re-binning (two kernels) and the step (two), not a list
    A.close()
    B.close()
