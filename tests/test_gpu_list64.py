"""FP64 sphere steps over the neighbour list (k_list64_step) against the oracle
and against the per-step path, bit for bit, with the per-step counters: slot
counts around the rule's limit and a block's 64, periodic and closed faces,
several colonies, crowds beyond a block's pair room and beyond a list's entries
(those states step on the per-step path), steps that leave the list's range, and
changes of the form between calls."""
import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, configs
from boltzmannmfx_gb300.abi import BMXG_ERR_NONFINITE, BMXG_FP32F, BMXG_FP64, Geometry
from boltzmannmfx_gb300.runtime import BmxgError

pytestmark = pytest.mark.gpu

OUT = ("x", "y", "z", "velx", "vely", "velz")
COUNTERS = ("n_out_of_domain", "n_edge_ghost", "n_pairs_last")
PRM = configs.deck_params()


def box(side, per, nz=32):
    m = int(round(side / configs.BIN))
    return Geometry.make((0.0, 0.0, 0.0), (side, side, nz * configs.BIN), (m, m, nz), (per, per, 0))


def colony(n, side, crowd, seed, z=0.045, spread=4.0e-4):
    P = configs.sphere_colony(n, side, side, np.random.default_rng(seed))
    rng = np.random.default_rng(seed + 1)
    for k, c in (("x", 0.0110), ("y", 0.0110), ("z", z)):
        P[k][:crowd] = c + rng.uniform(-spread, spread, crowd)
    return P


def join(parts):
    if len(parts) == 1:
        return parts[0]
    P = type(parts[0])(sum(p.n for p in parts))
    for k in P.a:
        P.a[k][...] = np.concatenate([p.a[k] for p in parts])
    return P


def state(ctx, P):
    Q = P.copy()
    ctx.get_state(Q)
    return Q


def same(A, B, P):
    QA, QB = state(A, P), state(B, P)
    for k in OUT:
        assert np.array_equal(QA[k], QB[k]), k
    sa, sb = A.stats(), B.stats()
    for k in COUNTERS:
        assert sa[k] == sb[k], k


@pytest.mark.parametrize("sizes, side, crowd, per", [
    ((16385,), 0.184, 0, 1), ((16448,), 0.184, 60, 0), ((16511,), 0.184, 300, 1), ((20011,), 0.184, 20, 1),
    ((15999, 1, 4000), 0.184, 22, 1), ((64, 16384), 0.184, 50, 0)])
def test_list_steps_equal_per_step_path(gpu_lib, oracle_lib, sizes, side, crowd, per):
    n = sum(sizes)
    geoms = [box(side, per) for _ in sizes]
    off = np.cumsum((0,) + sizes)
    P = join([colony(m, side, min(crowd, m), m) for m in sizes])
    A, B = Context(PRM, geoms), Context(PRM, geoms)
    B.set_list_mode(0)
    for c in (A, B):
        c.set_state(P, off)
        c.step(0.25, 160, BMXG_FP64)  # (enough steps for the rule to take the list)
    same(A, B, P)
    over = crowd > 32  # some list overflows: one build, then the per-step path
    assert (A.stats()["n_rebins"] == 161 if over else A.stats()["n_rebins"] < 160)
    assert B.stats()["n_rebins"] == 160
    for k in (3, 1, 9):
        A.step(0.25, k, BMXG_FP64)
        B.step(0.25, k, BMXG_FP64)
        same(A, B, P)
    # new inputs of the same size: the crowd is dense again, and the oracle's steps
    A.set_state(P, off)
    r0 = A.stats()["n_rebins"]
    A.step(0.25, 6, BMXG_FP64)
    assert (A.stats()["n_rebins"] - r0 == 7 if over else A.stats()["n_rebins"] - r0 < 6)
    R = P.copy()
    oracle_lib.evolve(PRM, geoms, off, R, 0.25, 6)
    Q = state(A, P)
    for k in OUT:
        assert np.array_equal(Q[k], R[k]), k
    pa = A.pairs()
    A.set_state(Q, off)
    for x, y in zip(pa, A.pairs()):
        assert np.array_equal(x, y)
    A.close()
    B.close()


def test_range_left_in_mid_call(gpu_lib):
    """A crowd above the domain's top passes the height the list covers within a
    call: the rest of the call runs on the per-step path."""
    n, side = 16500, 0.184
    g = [box(side, 1, 3)]
    P = configs.sphere_colony(n, side, side, np.random.default_rng(5))
    P["z"][...] = np.random.default_rng(6).uniform(0.001, 0.005, n)
    warm = P.copy()
    rng = np.random.default_rng(7)
    top = 1.7 * 3 * configs.BIN - 3.0e-5
    for k, c in (("x", 0.011), ("y", 0.011)):
        P[k][:20] = c + rng.uniform(-2.0e-4, 2.0e-4, 20)
    P["z"][:20] = top - rng.uniform(0.0, 4.0e-4, 20)
    A, B = Context(PRM, g), Context(PRM, g)
    B.set_list_mode(0)
    A.set_state(warm)
    A.step(0.25, 160, BMXG_FP64)
    for c in (A, B):
        c.set_state(P)
    r0 = A.stats()["n_rebins"]
    A.step(0.25, 20, BMXG_FP64)
    B.step(0.25, 20, BMXG_FP64)
    same(A, B, P)
    assert A.stats()["n_out_of_domain"] > 0
    assert state(A, P)["z"].max() > 1.7 * 3 * configs.BIN
    assert 2 < A.stats()["n_rebins"] - r0 < 20
    # from the start out of range: all of it per step
    A.step(0.25, 10, BMXG_FP64)
    B.step(0.25, 10, BMXG_FP64)
    same(A, B, P)
    A.close()
    B.close()


def test_form_changes_between_calls(gpu_lib):
    n, side = 16700, 0.184
    g = [box(side, 1)]
    P = colony(n, side, 20, 11)
    A, B = Context(PRM, g), Context(PRM, g)
    B.set_list_mode(0)
    A.set_state(P)
    A.step(0.25, 160, BMXG_FP64)
    A.step(0.25, 8, BMXG_FP32F)
    B.set_state(state(A, P))
    A.step(0.25, 7, BMXG_FP64)
    B.step(0.25, 7, BMXG_FP64)
    same(A, B, P)
    A.set_list_mode(0)
    A.step(0.25, 3, BMXG_FP64)
    A.set_list_mode(1)
    A.step(0.25, 9, BMXG_FP64)
    B.step(0.25, 12, BMXG_FP64)
    same(A, B, P)
    A.close()
    B.close()


@pytest.mark.parametrize("nsteps", [5, 40])
def test_prepared_and_profiled_calls(gpu_lib, nsteps):
    """The steps launched one by one (profiling) and as graphs are the same."""
    n, side = 16640, 0.184
    g = [box(side, 0)]
    P = colony(n, side, 20, 13)
    A, B = Context(PRM, g), Context(PRM, g)
    for c in (A, B):
        c.set_state(P)
        c.step(0.25, 160, BMXG_FP64)
        c.set_state(P)
    A.prepare(0.25, BMXG_FP64)
    B.set_profiling(True)
    A.step(0.25, nsteps, BMXG_FP64)
    B.step(0.25, nsteps, BMXG_FP64)
    same(A, B, P)
    A.close()
    B.close()


@pytest.mark.parametrize("field, bad", [("x", np.nan), ("y", -np.inf), ("z", np.inf)])
def test_non_finite_positions_are_reported(gpu_lib, field, bad):
    n, side = 16640, 0.184
    g = [box(side, 0)]
    P = colony(n, side, 0, 17)
    N = P.copy()
    N[field][n // 2] = bad
    A, B = Context(PRM, g), Context(PRM, g)
    B.set_list_mode(0)
    for c in (A, B):
        c.set_state(P)
        c.step(0.25, 160, BMXG_FP64)
        c.set_state(N)
        with pytest.raises(BmxgError) as e:
            c.step(0.25, 8, BMXG_FP64)
        assert e.value.code == BMXG_ERR_NONFINITE
        c.set_state(P)
        c.step(0.25, 8, BMXG_FP64)
    same(A, B, P)
    A.close()
    B.close()
