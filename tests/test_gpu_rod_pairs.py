"""The FP64 rod step over recorded pairs (k_rod_book queues every gated pair, one
per thread evaluates it, a segment adds its pairs in list order) at the sizes
where it can go wrong: one segment, a warp and one more, a block's tail, and
segments with more gated pairs than the lists hold (those walk the stencil),
alone and beside segments with few."""
import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, configs
from boltzmannmfx_gb300.abi import BMXG_FP64
from oracle import oracle as O

from common import trig_floor, within

pytestmark = pytest.mark.gpu


def segments(n, clump, seed):
    """n segments of seeded trees; the first `clump` of them moved within a fifth
    of a bin of one point, so that each is inside the gate of all the others."""
    per = max(1, min(n, 100))
    w = configs.rod_trees(seed=seed, ntrees=(n + per - 1) // per, per_tree=per, lx=0.064, ly=0.064)
    P = w.particles.subset(0, n)
    rng = np.random.default_rng(seed)
    for k, c in (("x", 0.0302), ("y", 0.0302), ("z", 0.0462)):
        P[k][:clump] = c + rng.uniform(0.0, 4.0e-4, clump)
    return w.params, w.geoms[0], P, w.dt


@pytest.mark.parametrize("n, clump", [(1, 0), (2, 2), (31, 0), (33, 33), (32, 32), (64, 34), (65, 20), (300, 60)])
def test_fp64_rod_step_over_recorded_pairs(gpu_lib, n, clump):
    prm, g, P, dt = segments(n, clump, 11 + n)
    pl = O.pairs(prm, g, P)
    R = P.copy()
    fc = O.forces(prm, g, R, pl)
    fv, fw = trig_floor(O, prm, g, P)
    ctx = Context(prm, [g])
    ctx.set_state(P)
    ctx.step(dt, 1, BMXG_FP64)
    Q = P.copy()
    ctx.get_state(Q)
    ctx.close()
    for c, k in enumerate(("velx", "vely", "velz")):
        assert within(Q[k], fc[c], 1.0e-10, 8 * fv + 1.0e-10 * np.abs(fc[:3]).max()), k
    for c, k in enumerate(("wx", "wy", "wz")):
        assert within(Q[k], fc[3 + c], 1.0e-10, 8 * fw + 1.0e-10 * np.abs(fc[3:]).max()), k
