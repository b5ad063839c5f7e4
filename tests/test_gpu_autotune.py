"""After bmxg_autotune the bins are the reference's for whatever comes next: the FP64
steps, the neighbour list and the FP32F per-step path of a tuned context are those
of an untuned one."""
import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, configs
from boltzmannmfx_gb300.abi import BMXG_FP32F, BMXG_FP64

pytestmark = pytest.mark.gpu

OUT = ("x", "y", "z", "velx", "vely", "velz")
PRM = configs.deck_params()


def loaded(n, side, seed):
    g = configs.box_geometry(side, side)
    P = configs.sphere_colony(n, side, side, np.random.default_rng(seed))
    ctx = Context(PRM, [g])
    ctx.set_state(P)
    return ctx, g, P


def read(ctx, P):
    Q = P.copy()
    ctx.get_state(Q)
    return Q


@pytest.mark.parametrize("then", ["step", "pairs", "forward", "fp32f"])
def test_first_call_after_autotune(gpu_lib, oracle_lib, then):
    n = 5000
    A, g, P = loaded(n, 0.064, 41)
    B, _, _ = loaded(n, 0.064, 41)
    A.autotune()
    if then == "pairs":
        assert all(np.array_equal(x, y) for x, y in zip(A.pairs(), B.pairs()))
        assert all(np.array_equal(x, y) for x, y in zip(A.pairs(), oracle_lib.pairs(PRM, g, P)))
    elif then == "forward":
        for c in (A, B):
            c.forward(0.25, 3, 2)
    else:
        for c in (A, B):
            if then == "fp32f":
                c.set_list_mode(0)
            c.step(0.25, 3, BMXG_FP32F if then == "fp32f" else BMXG_FP64)
    QA, QB = read(A, P), read(B, P)
    for k in OUT if then != "pairs" else OUT[:3]:
        assert np.array_equal(QA[k], QB[k]), k
    A.close()
    B.close()


def cached(path, n, side, **shape):
    """A tuning file whose FP64 sphere entry is replaced."""
    import json
    ctx, _, _ = loaded(n, side, 43)
    ctx.autotune(str(path))
    ctx.close()
    d = json.loads(path.read_text())
    key, = [k for k in d if "|sphere" in k and "|0|" in k]
    d[key].update(shape)
    path.write_text(json.dumps(d, separators=(", ", ": ")))
    return d, key


def test_a_tuned_sphere_shape_leaves_the_adjoint_its_kernels(gpu_lib, tmp_path):
    """The adjoint's kernels are chosen by its own rule, not by the grid that the
    tuning found for the FP64 step (one thread per slot takes twice as long here)."""
    import time
    n, side = 20_000, 0.128
    cached(tmp_path / "t.json", n, side, block=64, grid=4864)
    grad = np.random.default_rng(2).normal(0.0, 1.0, (3, n))
    best, got = [], []
    for tuned in (True, False):
        ctx, _, P = loaded(n, side, 43)
        if tuned:
            ctx.autotune(str(tmp_path / "t.json"))
            assert ctx.shapes()["sphere_grid"][0] == 4864
            ctx.set_shapes(list_step_passes=1)  # (the others as they are)
        t = []
        for _ in range(8):
            ctx.set_state(P)
            a = time.perf_counter()
            ctx.forward(0.25, 20, 10)
            out = ctx.backward(grad)
            t.append(time.perf_counter() - a)
        got.append(out)
        best.append(min(t[2:]))
        ctx.close()
    for x, y in zip(*got):
        assert np.array_equal(x, y)
    assert best[0] < 1.4 * best[1]


def test_entries_of_other_kernels_are_timed_again(gpu_lib, tmp_path):
    import json
    n, side = 2000, 0.064
    path = tmp_path / "t.json"
    d, key = cached(path, n, side)
    old = {k.replace("|sphere 2|", "|sphere|").replace("|list 2|", "|list|"): v for k, v in d.items()}
    assert not set(old) & set(d)
    for k in old:
        if "|sphere|0|" in k:
            old[k] = {"block": 96, "grid": 4097, "ms_per_5": 0.0}
    path.write_text(json.dumps(old, separators=(", ", ": ")))
    ctx, _, _ = loaded(n, side, 43)
    ctx.autotune(str(path))
    assert ctx.shapes()["sphere_block"][0] != 96
    ctx.close()
    assert set(json.loads(path.read_text())) == set(old) | set(d)  # (the file keeps both)
