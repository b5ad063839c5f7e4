"""List steps whose builds fall due every step or every few (long time steps): the
graphs with a build possible before every step, in calls split in several ways, give
the results and the builds of steps launched one by one."""
import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, configs
from boltzmannmfx_gb300.abi import BMXG_FP32F

pytestmark = pytest.mark.gpu

OUT = ("x", "y", "z", "velx", "vely", "velz")


@pytest.mark.parametrize("dt", [2.0, 8.0])
@pytest.mark.parametrize("calls", [(40,), (3, 37), (16, 1, 2, 21), (8, 8, 8, 8, 8), (5, 13, 22)])
def test_frequent_builds(gpu_lib, dt, calls):
    n, side = 3000, 0.064
    prm, g = configs.deck_params(), configs.box_geometry(side, side)
    P = configs.sphere_colony(n, side, side, np.random.default_rng(3))
    A, B = Context(prm, [g]), Context(prm, [g])
    B.set_profiling(True)  # (launched one by one)
    for _ in range(2):     # (the second time the period is known)
        for c in (A, B):
            c.set_state(P)
            r0 = c.stats()["n_rebins"]
            for k in calls:
                c.step(dt, k, BMXG_FP32F)
            c.builds = c.stats()["n_rebins"] - r0
        assert A.builds == B.builds >= 40 / (4.5 if dt < 8.0 else 2.0)
        QA, QB = P.copy(), P.copy()
        A.get_state(QA)
        B.get_state(QB)
        for k in OUT:
            assert np.array_equal(QA[k], QB[k]), k
    A.close()
    B.close()
