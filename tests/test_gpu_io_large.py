"""Device arrays of states whose fields together are more than one pass scatters (or, with
velocities, gathers): every field stored at once is the field stored alone, for FP64
positions, the list's fixed point, FP32F velocities and segments; velocities loaded
with the positions come back."""
import ctypes as C

import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, abi, configs
from boltzmannmfx_gb300.abi import BMXG_DEVICE, BMXG_FP32F, BMXG_FP64

pytestmark = pytest.mark.gpu

PRM = configs.deck_params()
SPHERE = ("x", "y", "z", "velx", "vely", "velz", "wx", "wy", "wz")
ROD = SPHERE + ("theta", "phi", "n_bnds", "seg_id1", "seg_id2", "site", "position", "fix_site", "fuse_flag",
                "split_flag", "new_flag", "dltd")


def struct(n, arrays):
    s = abi.ParticlesStruct()
    s.n = n
    for name, ctype in abi.ParticlesStruct._fields_[1:]:
        t = arrays.get(name)
        setattr(s, name, C.cast(C.c_void_p(t.data_ptr()), ctype) if t is not None else ctype())
    return s


def stored(ctx, n, fields):
    import torch
    out = {f: torch.zeros(n * abi.PLANE_FIELDS.get(f, 1), device="cuda",
                          dtype=torch.int32 if f in abi.INT_FIELDS or f in abi.PLANE_FIELDS else torch.float64)
           for f in fields}
    rc = ctx.lib.bmxg_get_state(ctx.h, C.byref(struct(n, out)), BMXG_DEVICE)
    assert rc == 0
    return {f: t.cpu().numpy() for f, t in out.items()}


def together_is_alone(ctx, n, fields):
    whole = stored(ctx, n, fields)
    for f in fields:
        assert np.array_equal(whole[f], stored(ctx, n, (f,))[f]), f
    return whole


def test_spheres(gpu_lib):
    import torch
    n, side = 1_210_007, 1.26
    g = configs.box_geometry(side, side)
    P = configs.sphere_colony(n, side, side, np.random.default_rng(91))
    for k, f in enumerate(SPHERE[3:]):
        P[f][...] = np.random.default_rng(k).normal(0.0, 1.0, n)
    dev = {f: torch.from_numpy(np.ascontiguousarray(P[f])).cuda() for f in SPHERE + ("radius", "cell_type")}
    torch.cuda.synchronize()
    ctx = Context(PRM, [g])
    assert ctx.lib.bmxg_set_state(ctx.h, C.byref(struct(n, dev)), None, BMXG_DEVICE) == 0
    ctx.n = n
    whole = together_is_alone(ctx, n, SPHERE)
    for f in SPHERE:
        assert np.array_equal(whole[f], P[f]), f
    ctx.step(0.25, 1, BMXG_FP64)
    together_is_alone(ctx, n, SPHERE)
    ctx.step(0.25, 3, BMXG_FP32F)
    a = together_is_alone(ctx, n, SPHERE)
    # the host's path, field by field
    Q = P.copy()
    ctx.get_state(Q, SPHERE)
    for f in SPHERE:
        assert np.array_equal(a[f], Q[f]), f
    ctx.close()


def test_rods(gpu_lib):
    """440 000 segments: copies of a few trees, one colony each."""
    trees, copies = 5, 880
    w = configs.rod_trees(ntrees=trees, per_tree=100, lx=0.064, ly=0.064)
    one = w.particles
    P = abi.Particles.concat([one] * copies)
    n = P.n
    off = np.arange(copies + 1, dtype=np.int64) * one.n
    ctx = Context(PRM, [configs.box_geometry(0.064, 0.064)] * copies)
    ctx.set_state(P, off)
    ctx.step(configs.ROD_DT, 2, BMXG_FP64)
    whole = together_is_alone(ctx, n, ROD)
    for f in ROD:  # the colonies are alike
        v = whole[f].reshape(abi.PLANE_FIELDS.get(f, 1), copies, one.n)
        assert np.array_equal(v, np.broadcast_to(v[:, :1], v.shape)), f
    ctx.close()
