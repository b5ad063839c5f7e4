"""Calls whose optional buffers find no room (bmxg_set_scratch_limit): FP64 sphere
steps without the list, FP64 rod steps that walk the stencil (k_rod_book_plain,
k_rod_force, k_rod_update) and the reverse sweep that bins each step's positions again
give the results of the paths with the buffers, bit for bit, and take them once
there is room."""
import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, abi, configs
from boltzmannmfx_gb300.abi import BMXG_FP64

pytestmark = pytest.mark.gpu

PRM = configs.deck_params()


def state(ctx, P):
    Q = P.copy()
    ctx.get_state(Q)
    return Q


def same(QA, QB):
    for k in QA.a:
        assert np.array_equal(QA.a[k], QB.a[k]), k


def test_fp64_list(gpu_lib):
    n, side = 30_000, 0.256
    g, P = configs.box_geometry(side, side), configs.sphere_colony(n, side, side, np.random.default_rng(51))
    A, B = Context(PRM, [g]), Context(PRM, [g])
    A.set_scratch_limit(1_000_000)
    for c in (A, B):
        c.set_state(P)
        c.step(0.25, 40, BMXG_FP64)
    assert A.stats()["n_rebins"] == 40 > B.stats()["n_rebins"]
    same(state(A, P), state(B, P))
    A.set_scratch_limit(-1)
    r0 = A.stats()["n_rebins"]
    for c in (A, B):
        c.step(0.25, 40, BMXG_FP64)
    assert A.stats()["n_rebins"] - r0 < 40
    same(state(A, P), state(B, P))
    A.close()
    B.close()


def rods(trees, spheres, crowd, seed):
    side = 0.128
    w = configs.rod_trees(seed=seed, ntrees=trees, per_tree=60, lx=side, ly=side)
    P = w.particles
    rng = np.random.default_rng(seed)
    # touching segments: more pairs at one than the queues hold
    for k, c in (("x", 0.0110), ("y", 0.0110), ("z", 0.0450)):
        P[k][:crowd] = c + rng.uniform(-4.0e-4, 4.0e-4, crowd)
    if spheres:
        S = configs.sphere_colony(spheres, side, side, rng)
        Q = abi.Particles(spheres, rods=True)
        for k in S.a:
            Q.a[k][...] = S.a[k]
        Q["id"] = np.arange(10_000_000, 10_000_000 + spheres)
        P = abi.Particles.concat([P, Q])
    return [configs.box_geometry(side, side)], P


@pytest.mark.parametrize("trees, spheres, crowd", [(1, 0, 0), (40, 0, 0), (20, 0, 50), (20, 900, 0)])
def test_fp64_rods(gpu_lib, trees, spheres, crowd):
    g, P = rods(trees, spheres, crowd, 53 + trees)
    A, B = Context(PRM, g), Context(PRM, g)
    A.set_scratch_limit(0)
    for c in (A, B):
        c.set_state(P)
    for steps in (1, 2, 9, 13):
        for c in (A, B):
            c.step(configs.ROD_DT, steps, BMXG_FP64)
        same(state(A, P), state(B, P))
        assert A.stats()["n_bond_repairs"] == B.stats()["n_bond_repairs"]
    A.set_scratch_limit(-1)   # the queues' steps on what the walk left
    for c in (A, B):
        c.step(configs.ROD_DT, 5, BMXG_FP64)
    same(state(A, P), state(B, P))
    A.close()
    B.close()


@pytest.mark.parametrize("n, steps, every", [(700, 7, 3), (4000, 12, 4), (4000, 5, 9), (300, 1, 1)])
def test_reverse_sweep(gpu_lib, n, steps, every):
    side = 0.064
    g, P = configs.box_geometry(side, side), configs.sphere_colony(n, side, side, np.random.default_rng(n))
    rng = np.random.default_rng(n + 1)
    adh, grad = rng.uniform(0.0, 1.0e-3, n), rng.normal(0.0, 1.0, (3, n))
    got = []
    for limit in (0, -1):
        ctx = Context(PRM, [g])
        ctx.set_scratch_limit(limit)
        ctx.set_state(P)
        ctx.set_ext(0.05, 1.0e-2, adh)
        ctx.forward(0.25, steps, every)
        out = list(ctx.backward(grad))
        out += list(ctx.backward(2.0 * grad))  # (again from the same trajectory)
        Q = state(ctx, P)
        ctx.step(0.25, 2, BMXG_FP64)           # and on from its end
        R = state(ctx, P)
        got.append(out + [Q[k] for k in "xyz"] + [R[k] for k in ("x", "y", "z", "velx", "vely", "velz")])
        ctx.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)


def test_a_sweep_gives_its_states_back(gpu_lib):
    """The kept states (here 460 MB) are not held after the sweep; another may follow."""
    import torch
    n, side, steps = 100_000, 0.384, 60
    g, P = configs.box_geometry(side, side), configs.sphere_colony(n, side, side, np.random.default_rng(61))
    grad = np.random.default_rng(62).normal(0.0, 1.0, (3, n))
    ctx = Context(PRM, [g])
    ctx.set_state(P)
    ctx.forward(0.25, steps, steps)
    ctx.step(0.25, 0, BMXG_FP64)
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    a = ctx.backward(grad)
    free1 = torch.cuda.mem_get_info()[0]
    assert free0 - free1 < 256 << 20
    for x, y in zip(a, ctx.backward(grad)):
        assert np.array_equal(x, y)
    ctx.close()
