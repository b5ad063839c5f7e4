"""Loads and stores in one pass, and the AoS records in place: device arrays
against host arrays (which go through the staging), aligned against misaligned
fields, host stores on both sides of the size where the fused kernel gives way
to the pipelined copies, positions straight from the list's fixed point, and AoS
records read in place against records staged whole."""
import ctypes as C

import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, abi, configs
from boltzmannmfx_gb300.abi import BMXG_DEVICE, BMXG_FP32F, BMXG_FP64, FUNGI, YEAST

pytestmark = pytest.mark.gpu

ROD_OUT = ("x", "y", "z", "theta", "phi", "velx", "vely", "velz", "wx", "wy", "wz", "n_bnds", "seg_id1", "seg_id2",
           "site", "position", "fix_site", "fuse_flag", "split_flag", "new_flag", "dltd")
OUT = ("x", "y", "z", "velx", "vely", "velz", "wx", "wy", "wz")


def device(P, fields, shift=0):
    """A struct of device copies of the fields; shift: bytes off a 16-byte boundary
    for every field but the five a load reads in place."""
    import torch
    s, keep = abi.ParticlesStruct(), {}
    s.n = P.n
    for name, ctype in abi.ParticlesStruct._fields_[1:]:
        if name not in fields:
            setattr(s, name, ctype())
            continue
        a = np.ascontiguousarray(P[name])
        off = 0 if name in ("x", "y", "z", "radius", "cell_type") else shift
        t = torch.zeros(a.nbytes + 16, dtype=torch.uint8, device="cuda")
        t[off:off + a.nbytes] = torch.from_numpy(a.view(np.uint8)).cuda()
        keep[name] = (t, off, a)
        setattr(s, name, C.cast(C.c_void_p(t.data_ptr() + off), ctype))
    torch.cuda.synchronize()
    return s, keep


def back(keep):
    return {k: t[off:off + a.nbytes].cpu().numpy().view(a.dtype) for k, (t, off, a) in keep.items()}


@pytest.mark.parametrize("trees, per, shift, vel", [(1, 1, 0, False), (3, 11, 0, True), (13, 80, 0, True),
                                                    (3, 43, 2, True), (700, 100, 0, False)])
def test_rods_device_arrays_equal_host_arrays(gpu_lib, trees, per, shift, vel):
    w = configs.rod_trees(seed=trees, ntrees=trees, per_tree=per, lx=0.512, ly=0.512)
    P = w.particles
    rng = np.random.default_rng(per)
    for k in ("fuse_tip", "fix_site", "fuse_flag"):
        P[k] = rng.integers(0, 3, P.n)
    P["dltd"] = rng.integers(-1, 5, 6 * P.n)
    fields = [f for f, _ in abi.ParticlesStruct._fields_[1:] if vel or f[:3] != "vel"]
    if not vel:
        fields.remove("bond_scale")
        fields.remove("dltd")
    got = []
    for dev in (False, True):
        ctx = Context(w.params, w.geoms)
        if dev:
            s, keep = device(P, fields, shift)
            assert ctx.lib.bmxg_set_state(ctx.h, C.byref(s), None, BMXG_DEVICE) == 0
            ctx.n = P.n
        else:
            ctx.set_state(P, fields=fields)
        ctx.step(w.dt, 2, BMXG_FP64)
        if dev:
            so, ko = device(P, ROD_OUT)
            assert ctx.lib.bmxg_get_state(ctx.h, C.byref(so), BMXG_DEVICE) == 0
            got.append(back(ko))
        else:
            Q = P.copy()
            ctx.get_state(Q, ROD_OUT)
            got.append({k: Q[k] for k in ROD_OUT})
        ctx.close()
    for k in ROD_OUT:
        assert np.array_equal(got[0][k], got[1][k]), k


@pytest.mark.parametrize("n", [1, 65536, 65537])
@pytest.mark.parametrize("prec, steps", [(BMXG_FP64, 1), (BMXG_FP32F, 3)])
def test_spheres_store_the_same_either_way(gpu_lib, n, prec, steps):
    """FP32F over three steps runs on the list: its positions are stored from the
    fixed point, in full or after only one axis was asked for."""
    side = 0.016 if n == 1 else 0.324
    P = configs.sphere_colony(n, side, side, np.random.default_rng(n))
    ctx = Context(configs.deck_params(), [configs.box_geometry(side, side)])
    ctx.set_state(P)
    ctx.step(0.25, steps, prec)
    so, ko = device(P, OUT)
    assert ctx.lib.bmxg_get_state(ctx.h, C.byref(so), BMXG_DEVICE) == 0
    ctx.set_state(P)
    ctx.step(0.25, steps, prec)
    A, B = P.copy(), P.copy()
    ctx.get_state(A, ("y",))
    ctx.get_state(A, OUT)
    ctx.set_state(P)
    ctx.step(0.25, steps, prec)
    ctx.get_state(B, OUT)
    ctx.close()
    dev = back(ko)
    for k in OUT:
        assert np.array_equal(A[k], B[k]), k
        assert np.array_equal(dev[k], B[k]), k


def records(P, spare=0):
    """P as AoS records, `spare` bytes into a buffer (a misaligned address is
    staged whole instead of read in place)."""
    buf = np.zeros(P.n * 448 + 16, np.uint8)
    off = (-buf.ctypes.data) % 16 + spare
    a = buf[off:off + P.n * 448].view(abi.aos_dtype()) if spare == 0 else None
    r = np.zeros(P.n, abi.aos_dtype())
    rng = np.random.default_rng(1)
    r["rdata"] = rng.normal(size=(P.n, 34))
    r["idata"] = rng.integers(0, 3, (P.n, 35))
    for d, f in enumerate(("x", "y", "z")):
        r["pos"][:, d] = P[f]
    for f in ("radius", "c_length", "theta", "phi", "area", "bond_scale"):
        r["rdata"][:, abi.REAL_IDX[f]] = P[f]
    for f in ("cell_type", "n_bnds", "position", "fuse_tip", "fix_site", "id", "cpu"):
        r["idata"][:, abi.INT_IDX[f]] = P[f]
    for f, base in (("seg_id1", 7), ("seg_id2", 11), ("site", 15)):
        r["idata"][:, base:base + 4] = P[f].reshape(4, P.n).T
    view = buf[off:off + P.n * 448]
    view[:] = r.view(np.uint8).reshape(-1)
    del a
    return buf, off, view


@pytest.mark.parametrize("kind", ["spheres", "rods", "rods_then_cells", "cells_then_rods"])
@pytest.mark.parametrize("n", [1, 127, 1000])
def test_aos_records_in_place_equal_staged(gpu_lib, kind, n):
    side = 0.128
    C0 = configs.sphere_colony(n, side, side, np.random.default_rng(n))
    if kind == "spheres":
        P = C0
    else:
        R0 = configs.rod_trees(seed=5, ntrees=1, per_tree=n, lx=side, ly=side).particles
        parts = {"rods": [R0], "rods_then_cells": [R0, C0], "cells_then_rods": [C0, R0]}[kind]
        P = abi.Particles.concat(parts)
        assert P["cell_type"][0] == (YEAST if kind == "cells_then_rods" else FUNGI)
    got = []
    for spare in (0, 4):
        buf, off, view = records(P, spare)
        ctx = Context(configs.deck_params(), [configs.box_geometry(side, side)])
        cost, nsub = (C.c_double * 1)(), C.c_int32(0)
        for _ in range(2):
            rc = ctx.lib.bmxg_evolve_particles_aos(ctx.h, C.c_void_p(buf.ctypes.data + off), P.n, 34, 35, None,
                                                   configs.ROD_DT, cost, C.byref(nsub))
            assert rc == 0, ctx.lib.bmxg_last_error(ctx.h)
        ctx.close()
        got.append(view.copy())
    assert np.array_equal(got[0], got[1])
    # and the SoA calls on the same state
    before = records(P)[2].view(abi.aos_dtype())
    after = got[0].view(abi.aos_dtype())
    same = np.ones(34, bool)
    same[[2, 3, 6, 7, 8, 9, 10, 11]] = False         # theta, phi, velx .. wz
    assert np.array_equal(before["rdata"][:, same], after["rdata"][:, same])
    Q = P.copy()
    ctx = Context(configs.deck_params(), [configs.box_geometry(side, side)])
    for _ in range(2):
        ctx.set_state(Q)
        ctx.step(configs.ROD_DT, 1, BMXG_FP64)
        ctx.get_state(Q, [f for f in ROD_OUT if f not in ("fuse_flag", "split_flag", "new_flag", "dltd")])
    ctx.close()
    for d, f in enumerate(("x", "y", "z")):
        assert np.array_equal(after["pos"][:, d], Q[f]), f
    for f in ("velx", "vely", "velz") + (("theta", "phi") if kind != "spheres" else ()):
        assert np.array_equal(after["rdata"][:, abi.REAL_IDX[f]], Q[f]), f
