"""The parameter gradients are sums over the slots in an order that the caller's order
moves: with pairs apart from one another every slot's own terms stay the same, and so
do the sums, to the last bit, since their roundings are kept beside them."""
import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, configs

pytestmark = pytest.mark.gpu


def test_order_of_the_slots(gpu_lib):
    m, side = 100, 0.064
    rng = np.random.default_rng(81)
    n = 2 * m * m
    g = configs.box_geometry(side, side)
    P = configs.sphere_colony(n, side, side, rng)
    P["radius"][...] = rng.uniform(1.0e-5, 1.5e-5, n)  # (cutoff 1.3e-4 at most)
    ix, iy = np.meshgrid(np.arange(m), np.arange(m), indexing="ij")
    for h in (0, 1):  # pairs 3e-4 apart, many in a bin, which the caller's order sorts
        P["x"][h::2] = (ix.ravel() + 0.5) * 3.0e-4 + rng.uniform(-2.0e-5, 2.0e-5, m * m)
        P["y"][h::2] = (iy.ravel() + 0.5) * 3.0e-4 + rng.uniform(-2.0e-5, 2.0e-5, m * m)
        P["z"][h::2] = 0.0450 + h * 8.0e-5
    adh, grad = rng.uniform(0.0, 1.0e-3, n), rng.normal(0.0, 1.0, (3, n))
    got = []
    for k in range(6):
        perm = rng.permutation(n) if k else np.arange(n)
        Q = P.copy()
        for f in ("x", "y", "z", "radius", "area"):
            Q[f][...] = P[f][perm]
        ctx = Context(configs.deck_params(), [g])
        ctx.set_state(Q)
        ctx.set_ext(0.05, 1.0e-2, adh[perm])
        ctx.forward(0.25, 1, 1)
        gx, gp, ga = ctx.backward(np.ascontiguousarray(grad[:, perm]))
        ctx.close()
        inv = np.argsort(perm)
        got.append((gx[:, inv], ga[inv], gp))
    assert np.all(got[0][2] != 0.0)
    for a in got[1:]:
        for x, y in zip(a, got[0]):
            assert np.array_equal(x, y)
