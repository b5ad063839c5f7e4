"""FP64 list steps of states loaded with positions beyond the periodic x and y
faces (a load does not wrap them, the first step does), against the per-step path,
bit for bit: a slot's images are the slots of the other face's bins, however near
the image of one farther in comes to a slot beyond the face.  (The oracle lists a
position's image that falls back into the box from the bin it is in; the library
counts it in n_edge_ghost.)"""
import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, configs
from boltzmannmfx_gb300.abi import BMXG_FP64, Geometry

pytestmark = pytest.mark.gpu

OUT = ("x", "y", "z", "velx", "vely", "velz")
PRM = configs.deck_params()


def beyond(n, side, pairs, far, seed):
    """A colony, its first 2 x pairs particles in pairs whose one is up to `far` beyond
    a face and whose other is that one's wrapped position plus less than the cutoff."""
    P = configs.sphere_colony(n, side, side, np.random.default_rng(seed))
    rng = np.random.default_rng(seed + 1)
    for q in range(pairs):
        ax, lo = ("x", "y")[q % 2], rng.random() < 0.5
        d = rng.uniform(0.0, far)
        i, j = 2 * q, 2 * q + 1
        P[ax][i] = -d if lo else side + d
        P[ax][j] = (side - d if lo else d) + rng.uniform(-1.2e-3, 1.2e-3)
        other = "y" if ax == "x" else "x"
        P[other][j] = P[other][i] + rng.uniform(-4.0e-4, 4.0e-4)
        P["z"][j] = P["z"][i] + rng.uniform(-4.0e-4, 4.0e-4)
        P["radius"][[i, j]] = 8.0e-4
    return P


@pytest.mark.parametrize("far", [1.0e-3, 5.0e-3, 0.05])
def test_positions_beyond_the_periodic_faces(gpu_lib, far):
    n, side = 16600, 0.184
    m = int(round(side / configs.BIN))
    g = [Geometry.make((0.0, 0.0, 0.0), (side, side, 0.064), (m, m, 32), (1, 1, 0))]
    P = beyond(n, side, 400, far, 23)
    A, B = Context(PRM, g), Context(PRM, g)
    B.set_list_mode(0)
    A.set_state(configs.sphere_colony(n, side, side, np.random.default_rng(29)))
    A.step(0.25, 160, BMXG_FP64)  # (the list's buffers are paid for)
    r0 = A.stats()["n_rebins"]
    for c in (A, B):
        c.set_state(P)
        c.step(0.25, 8, BMXG_FP64)
    assert A.stats()["n_rebins"] - r0 < 8  # over the list
    QA, QB = P.copy(), P.copy()
    A.get_state(QA)
    B.get_state(QB)
    for k in OUT:
        assert np.array_equal(QA[k], QB[k]), k
    A.close()
    B.close()
