"""Performance cases of the particle step: what a user's program has it do.

Every case goes through the public entry points (the C ABI of include/bmxg.h
by its ctypes binding).  Device-resident programs hand over their arrays as
device addresses and give the library the stream they run on; programs whose
particles are host data (AMReX's AoS tiles, host SoA arrays) hand over host
memory.  Each pass starts from the same loaded inputs, so passes repeat the
same work.  Velocities of the FP32F form come back in FP32, the precision that
form computes them in.
"""
import ctypes as C
import math

import numpy as np
import torch

from boltzmannmfx_gb300 import abi, configs, runtime
from boltzmannmfx_gb300.abi import BMXG_DEVICE, BMXG_FP32F, BMXG_FP64, FUNGI, YEAST

DT = 0.25                                  # time step of the sphere configurations
SPHERE_IN = ("x", "y", "z", "radius", "cell_type")
SPHERE_OUT = ("x", "y", "z", "velx", "vely", "velz")
ROD_IN = SPHERE_IN + ("c_length", "theta", "phi", "area", "bond_scale", "id", "cpu", "n_bnds", "seg_id1", "seg_id2",
                      "site", "position", "fuse_tip", "fix_site", "dltd")
ROD_OUT = ("x", "y", "z", "theta", "phi", "velx", "vely", "velz", "wx", "wy", "wz", "n_bnds", "seg_id1", "seg_id2",
           "site", "position")
PRECISION = {"fp64": BMXG_FP64, "fp32f": BMXG_FP32F}


# ---- the cases ---------------------------------------------------------------

def listed():
    return [
        # EvolveParticles on the reference's own records (the C++ shim's call, once per time step):
        # a network of the size of the shipped one, and a tile of yeast cells
        dict(name="aos_network_400", kind="aos", cells="rods", trees=5, per_tree=80),
        dict(name="aos_cells_20k", kind="aos", cells="spheres", n=20_011, side=0.128),
        # one AMReX tile (a quarter of the 0.128 cm level) with its ghosts, once per time step
        dict(name="tile_quarter_20k", kind="tile", n=20_000, cells=64, tile=32),
        # the plain form: a small colony over 100 steps, and many colonies at once
        dict(name="fp64_2k_100", kind="spheres", precision="fp64", colonies=1, n=2_000, side=0.128, steps=100),
        dict(name="fp64_colonies_64_10", kind="spheres", precision="fp64", colonies=64, nmin=500, nmax=50_000,
             side=0.128, steps=10),
        # the precision form: one mid-size domain, and the batched colonies
        dict(name="fp32f_200k_100", kind="spheres", precision="fp32f", colonies=1, n=200_000, side=0.512, steps=100),
        dict(name="fp32f_colonies_256_100", kind="spheres", precision="fp32f", colonies=256, nmin=500, nmax=50_000,
             side=0.128, steps=100),
        # EvolveParticles from host SoA arrays whose state changes between the calls (after chemistry and division)
        dict(name="host_fp64_500k", kind="host", n=499_979, side=0.768),
        # hyphal trees, both forms
        dict(name="rods_fp64_50k_10", kind="rods", precision="fp64", trees=500, per_tree=100, side=0.512, steps=10),
        dict(name="rods_fp32f_50k_20", kind="rods", precision="fp32f", trees=500, per_tree=100, side=0.512, steps=20),
        # the differentiation form: forward and backward over a checkpointed trajectory
        dict(name="adjoint_20k_40", kind="adjoint", n=20_000, side=0.128, steps=40, every=20),
        # split_particles after a step: a twentieth of the cells divide
        dict(name="split_500k", kind="split", n=500_000, share=0.05),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _bins(side):
    """A box side of whole bins."""
    return max(3, round(side / configs.BIN)) * configs.BIN


def draw(rng):
    kind = rng.choice(["aos", "tile", "spheres", "spheres", "spheres", "spheres", "host", "rods", "rods", "adjoint",
                       "split"])
    if kind == "aos":
        if rng.random() < 0.5:
            return dict(kind="aos", cells="rods", trees=_log(rng, 2, 60), per_tree=rng.randint(40, 100))
        n = _log(rng, 300, 60_000)
        return dict(kind="aos", cells="spheres", n=n, side=_bins(0.128 * max(0.25, math.sqrt(n / 20_000))))
    if kind == "tile":
        cells = rng.choice([32, 48, 64])
        return dict(kind="tile", n=_log(rng, 500, 40_000), cells=cells, tile=rng.randint(cells // 4, cells // 2))
    if kind == "spheres":
        precision = rng.choice(["fp64", "fp32f"])
        if rng.random() < 0.5:
            n = _log(rng, 500, 250_000)
            return dict(kind="spheres", precision=precision, colonies=1, n=n,
                        side=_bins(0.128 * max(0.5, math.sqrt(n / 12_500))), steps=rng.randint(8, 100))
        nmax = _log(rng, 2_000, 50_000)
        return dict(kind="spheres", precision=precision, colonies=rng.randint(2, 128), nmin=500, nmax=nmax,
                    side=rng.choice([0.096, 0.128, 0.162]),
                    steps=rng.randint(4, 12) if precision == "fp64" else rng.randint(8, 100))
    if kind == "host":
        n = _log(rng, 2_000, 900_000)
        return dict(kind="host", n=n, side=_bins(0.128 * max(0.5, math.sqrt(n / 12_500))))
    if kind == "rods":
        trees = _log(rng, 5, 500)
        return dict(kind="rods", precision=rng.choice(["fp64", "fp32f"]), trees=trees, per_tree=rng.randint(40, 100),
                    side=_bins(0.512 * max(0.25, math.sqrt(trees / 500))), steps=rng.randint(4, 20))
    if kind == "adjoint":
        n = _log(rng, 1_000, 40_000)
        return dict(kind="adjoint", n=n, side=_bins(0.128 * max(0.5, math.sqrt(n / 20_000))),
                    steps=rng.randint(10, 60), every=rng.choice([5, 10, 20]))
    return dict(kind="split", n=_log(rng, 2_000, 900_000), share=rng.choice([0.01, 0.05, 0.2]))


def work(case):
    """Bytes each pass cannot do without: the state read and written once per
    step (80 B per FP64 sphere, 64 B per FP32F sphere, 212 / 188 B per FP64 /
    FP32F segment), plus the load and the store; for a division the decision's
    12 B per record and 968 B per new particle."""
    k = case["kind"]
    if k == "split":
        new = case["n"] * case["share"]
        return {"bytes": 12.0 * case["n"] + 968.0 * new, "flops": 100.0 * new}
    if k == "aos":
        rods = case["cells"] == "rods"
        n = _size(case)
        return {"bytes": n * ((36 + 48.0 + 80) if not rods else (172 + 160 + 212.0)),
                "flops": n * (1500.0 if rods else 120.0)}
    if k == "tile":
        n = _tile_own(case)
        return {"bytes": 80.0 * n, "flops": 120.0 * n}
    n = _size(case)
    if k == "host":
        return {"bytes": n * (36 + 48 + 80.0), "flops": 120.0 * n}
    if k == "adjoint":
        t = case["steps"]
        # forward, recomputation and reverse sweep
        return {"bytes": n * t * (80 + 80 + 128.0), "flops": n * t * 600.0}
    per = {"spheres": {"fp64": 80.0, "fp32f": 64.0}, "rods": {"fp64": 212.0, "fp32f": 188.0}}[k][case["precision"]]
    load = 84.0 if k == "spheres" else 340.0
    return {"bytes": n * (load + per * case["steps"]),
            "flops": n * case["steps"] * (100.0 if k == "spheres" else 1200.0)}


def _sizes(case):
    """Particles per colony: log-uniform sizes, the same ones for every seed."""
    c = case["colonies"]
    if c == 1:
        return [case["n"]]
    lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
    return [int(math.exp(lo + (hi - lo) * (q + 0.5) / c)) for q in range(c)]


def _size(case):
    if case["kind"] == "spheres":
        return sum(_sizes(case))
    if case["kind"] == "rods" or case.get("cells") == "rods":
        return case["trees"] * case["per_tree"]
    return case["n"]


# ---- inputs ------------------------------------------------------------------

def _spheres(n, side, seed):
    """Seeded spheres of the configurations' distributions, on the device."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + n)
    u = torch.rand((4, n), generator=g, dtype=torch.float64, device="cuda")
    zlo, zhi = configs.Z_BAND
    pos = torch.empty((3, n), dtype=torch.float64, device="cuda")
    pos[0] = u[0] * side
    pos[1] = u[1] * side
    pos[2] = zlo + u[2] * (zhi - zlo)
    return pos, 5.0e-4 + 3.0e-4 * u[3]


def _colony_order(case, seed):
    sizes = np.array(_sizes(case), np.int64)
    sizes = sizes[np.random.default_rng(seed).permutation(len(sizes))]
    off = np.zeros(len(sizes) + 1, np.int64)
    off[1:] = np.cumsum(sizes)
    return off


def _trees(trees, per_tree, side, seed):
    """Branching hyphal trees as configs.rod_trees draws them, every tree grown
    at once: a segment starts at the end of its parent (the tree's last segment,
    or an earlier one where it branches), bonded end to end."""
    rng = np.random.default_rng(seed)
    n = trees * per_tree
    row = np.arange(trees)
    X = np.zeros((trees, per_tree, 3))
    TH = np.zeros((trees, per_tree))
    PH = np.zeros((trees, per_tree))
    L = rng.uniform(30.0e-4, 35.0e-4, (trees, per_tree))
    tip = np.zeros((trees, per_tree, 3))
    nb = np.zeros((trees, per_tree), np.int32)
    ids = np.arange(1, n + 1, dtype=np.int32).reshape(trees, per_tree)
    s1 = np.zeros((4, trees, per_tree), np.int32)
    site = np.zeros((4, trees, per_tree), np.int32)
    child = np.zeros((trees, per_tree), bool)
    zlo, zhi = configs.Z_BAND
    root = np.stack([rng.uniform(0, side, trees), rng.uniform(0, side, trees),
                     rng.uniform(zlo + 0.002, zhi - 0.002, trees)], axis=1)
    root_ph = rng.uniform(0.0, 2.0 * np.pi, trees)
    for k in range(per_tree):
        th = rng.normal(0.0, 0.05, trees)
        ph = rng.normal(0.0, 0.15, trees)
        turn = np.radians(rng.uniform(30.0, 90.0, trees)) * np.where(rng.random(trees) < 0.5, 1.0, -1.0)
        if k == 0:
            start, th, ph = root, np.pi / 2 + th, root_ph + ph
        else:
            branch = rng.random(trees) < 0.05
            p = np.where(branch, rng.integers(0, k, trees), k - 1)
            p = np.where(nb[row, p] < 4, p, k - 1)
            start = tip[row, p]
            th = TH[row, p] + th
            ph = PH[row, p] + ph + np.where(branch, turn, 0.0)
            for a, b, w in ((np.full(trees, k), p, 1), (p, np.full(trees, k), 2)):
                m = nb[row, a]
                s1[m, row, a] = ids[row, b]
                site[m, row, a] = w
                nb[row, a] += 1
            child[row, p] = True
        th = np.clip(th, np.pi / 2 - 0.3, np.pi / 2 + 0.3)
        ph = ph % (2.0 * np.pi)
        half = 0.5 * L[:, k, None]
        ax = np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)], axis=1)
        c = start + half * ax
        out = (c[:, 2] < zlo + 0.001) | (c[:, 2] > zhi - 0.001)      # keep in the z band
        th = np.where(out, np.pi - th, th)
        ax[:, 2] = np.where(out, -ax[:, 2], ax[:, 2])
        X[:, k] = start + half * ax
        tip[:, k] = X[:, k] + half * ax
        TH[:, k], PH[:, k] = th, ph
    X = X.reshape(n, 3)
    X[:, :2] %= side
    P = abi.Particles(n, rods=True)
    P["x"], P["y"], P["z"] = X[:, 0], X[:, 1], X[:, 2]
    P["theta"], P["phi"], P["c_length"] = TH.reshape(n), PH.reshape(n), L.reshape(n)
    r = 2.0e-4
    P["radius"] = r
    P["area"] = 2.0 * math.pi * r * L.reshape(n) + 2.0 * math.pi * r * r
    P["cell_type"] = FUNGI
    P["id"] = ids.reshape(n)
    P["n_bnds"] = nb.reshape(n)
    P["seg_id1"] = s1.reshape(-1)
    P["site"] = site.reshape(-1)
    P["position"] = np.where(child, abi.SITE_INTERIOR, abi.SITE_TIP).reshape(n)
    return P


def _struct(n, fields):
    """bmxg_particles over device tensors."""
    s = abi.ParticlesStruct()
    s.n = n
    for name, ctype in abi.ParticlesStruct._fields_[1:]:
        t = fields.get(name)
        setattr(s, name, C.cast(C.c_void_p(t.data_ptr()), ctype) if t is not None else ctype())
    return s


class _Domain:
    """A device-resident program: a context on the program's stream, its input
    arrays and the arrays it reads the state back into."""

    def __init__(self, geoms, n, inputs, outputs, offsets=None):
        self.stream = torch.cuda.Stream()
        self.ctx = runtime.Context(configs.deck_params(), geoms)
        self.ctx.set_stream(self.stream.cuda_stream)
        self.inputs, self.outputs = inputs, outputs
        self.s_in, self.s_out = _struct(n, inputs), _struct(n, outputs)
        self.off = offsets
        self.off_ptr = None if offsets is None else offsets.ctypes.data_as(C.POINTER(C.c_int64))
        self.ctx.n = n
        torch.cuda.current_stream().synchronize()  # the inputs are made

    def check(self, rc):
        if rc:
            raise runtime.BmxgError(rc, self.ctx.lib.bmxg_last_error(self.ctx.h).decode())

    def load(self):
        self.check(self.ctx.lib.bmxg_set_state(self.ctx.h, C.byref(self.s_in), self.off_ptr, BMXG_DEVICE))

    def store(self):
        self.check(self.ctx.lib.bmxg_get_state(self.ctx.h, C.byref(self.s_out), BMXG_DEVICE))


def _planes(fields, rows):
    return {f: t for f, t in zip(fields, rows)}


def _records(P):
    """BMX's 448-byte records of a particle container."""
    a = np.zeros(P.n, abi.aos_dtype())
    for d, f in enumerate(("x", "y", "z")):
        a["pos"][:, d] = P[f]
    for f in ("radius", "c_length", "theta", "phi", "area", "bond_scale"):
        a["rdata"][:, abi.REAL_IDX[f]] = P[f]
    for f in ("cell_type", "n_bnds", "position", "fuse_tip", "fix_site", "id", "cpu"):
        a["idata"][:, abi.INT_IDX[f]] = P[f]
    for f, base, k in (("seg_id1", 7, 4), ("seg_id2", 11, 4), ("site", 15, 4), ("dltd", 26, 6)):
        a["idata"][:, base:base + k] = P[f].reshape(k, P.n).T
    a["id"], a["cpu"] = P["id"], P["cpu"]
    return a


def _aos_side(case):
    return case["side"] if case["cells"] == "spheres" else _bins(0.512 * max(0.25, math.sqrt(case["trees"] / 500)))


def _aos_particles(case, seed):
    if case["cells"] == "rods":
        return _trees(case["trees"], case["per_tree"], _aos_side(case), seed)
    pos, r = _spheres(case["n"], case["side"], seed)
    P = abi.Particles(case["n"])
    P["x"], P["y"], P["z"] = pos.cpu().numpy()
    P["radius"] = r.cpu().numpy()
    P["area"] = 4.0 * math.pi * P["radius"] ** 2
    P["cell_type"] = YEAST
    return P


def _tile_own(case):
    return max(1, round(case["n"] * (case["tile"] / case["cells"]) ** 2))


def _split_records(case, seed):
    n = case["n"]
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 104729 + n)

    def uni(*shape):
        return torch.rand(shape, generator=g, dtype=torch.float64, device="cuda")

    cap = n + int(n * case["share"] * 1.5) + 64
    rec = torch.zeros((cap, 56), dtype=torch.float64, device="cuda")
    rec[:n, 0:2] = uni(n, 2) * 0.128
    rec[:n, 2] = 0.04 + 0.012 * uni(n)
    rec[:n, 3:37] = uni(n, 34) - 0.5
    split = torch.zeros(n, dtype=torch.bool, device="cuda")
    split[torch.randperm(n, generator=g, device="cuda")[:max(1, int(n * case["share"]))]] = True
    vol = 5.0e-10 * torch.where(split, 1.0001 + 0.9 * uni(n), 0.4 + 0.6 * uni(n))
    R = abi.REAL_IDX
    radius = (3.0 * vol / (4.0 * math.pi)) ** (1.0 / 3.0)
    rec[:n, 3 + R["vol"]] = vol
    rec[:n, 3 + R["radius"]] = radius
    rec[:n, 3 + R["area"]] = 4.0 * math.pi * radius * radius
    rec[:n, 3 + R["dvdt"]] = 1.0e-12 * uni(n)
    ints = rec.view(torch.int32)                       # ids at 74, 75; idata from 76
    ids = torch.arange(1, n + 1, dtype=torch.int32, device="cuda")
    ints[:n, 74] = ids
    ints[:n, 76 + abi.INT_IDX["id"]] = ids
    ints[:n, 76 + abi.INT_IDX["cell_type"]] = YEAST
    mothers = torch.nonzero(split).reshape(-1)
    draws = uni(2 * mothers.numel() + 2)
    return rec, mothers, draws


def _tile_inputs(case, seed):
    """The tile's own particles (the share of the level's that its area has) and
    the copies of the others within one cell of it."""
    nc, tl = case["cells"], case["tile"]
    side, edge = nc * configs.BIN, tl * configs.BIN
    n_own = _tile_own(case)
    pos, r = _spheres(case["n"], side, seed)
    # the first n_own inside the tile, the others in the level's remaining L: the strip beside the tile, or above it
    pos[:2, :n_own] *= edge / side
    x, y = pos[0, n_own:] / side, pos[1, n_own:]
    beside = side * (side - edge) / (side * side - edge * edge)
    strip = x < beside
    pos[0, n_own:] = torch.where(strip, edge + x / beside * (side - edge), (x - beside) / (1.0 - beside) * edge)
    pos[1, n_own:] = torch.where(strip, y, edge + y * (1.0 - edge / side))
    nz = 32
    inv = [1.0 / (side / nc), 1.0 / (side / nc), 1.0 / (0.064 / nz)]
    cell = [torch.floor(pos[d] * inv[d]).long().clamp(0, (nc, nc, nz)[d] - 1) for d in range(3)]
    own = torch.arange(case["n"], device="cuda") < n_own
    # (rounding at the tile's edge: back inside)
    for d in range(2):
        pos[d] = torch.where(own & (cell[d] >= tl), torch.full_like(pos[d], edge * (1.0 - 1.0e-9)), pos[d])
        cell[d] = torch.floor(pos[d] * inv[d]).long().clamp(0, nc - 1)
    parts = []
    for sx in (-1, 0, 1):
        for sy in (-1, 0, 1):
            px, py = pos[0] + sx * side, pos[1] + sy * side
            cx = torch.floor(px * inv[0]).long() if sx else cell[0]
            cy = torch.floor(py * inv[1]).long() if sy else cell[1]
            near = (cx >= -1) & (cx <= tl) & (cy >= -1) & (cy <= tl)
            sel = torch.nonzero(near & ~((cx < tl) & (cy < tl) & (cx >= 0) & (cy >= 0))).reshape(-1)
            parts.append((sel, px[sel], py[sel]))
    idx = torch.cat([p[0] for p in parts])
    order = torch.argsort(idx, stable=True)
    idx = idx[order]
    ghosts = torch.stack([torch.cat([p[1] for p in parts])[order], torch.cat([p[2] for p in parts])[order],
                          pos[2][idx]]).contiguous()
    return pos[:, :n_own].contiguous(), r[:n_own].contiguous(), ghosts, r[idx].contiguous()


def prepare(case, seed):
    k = case["kind"]
    S = dict(case=case)
    if k == "spheres":
        off = _colony_order(case, seed)
        n = int(off[-1])
        pos, r = _spheres(n, case["side"], seed)
        out = torch.empty((6, n), dtype=torch.float64, device="cuda")
        inputs = dict(x=pos[0], y=pos[1], z=pos[2], radius=r,
                      cell_type=torch.full((n,), YEAST, dtype=torch.int32, device="cuda"))
        geoms = [configs.box_geometry(case["side"], case["side"])] * case["colonies"]
        S.update(dom=_Domain(geoms, n, inputs, _planes(SPHERE_OUT, out), off if case["colonies"] > 1 else None),
                 out=out)
    elif k == "rods":
        P = _trees(case["trees"], case["per_tree"], case["side"], seed)
        inputs = {f: torch.from_numpy(np.ascontiguousarray(P[f])).cuda() for f in ROD_IN}
        planes = {f: (abi.PLANE_FIELDS.get(f, 1), torch.int32 if f in abi.INT_FIELDS or f in abi.PLANE_FIELDS
                      else torch.float64) for f in ROD_OUT}
        out = {f: torch.empty(m * P.n, dtype=d, device="cuda") for f, (m, d) in planes.items()}
        S.update(dom=_Domain([configs.box_geometry(case["side"], case["side"])], P.n, inputs, out), out=out)
    elif k == "aos":
        side = _aos_side(case)
        rec = _records(_aos_particles(case, seed))
        S.update(ctx=runtime.Context(configs.deck_params(), [configs.box_geometry(side, side)]), start=rec,
                 rec=rec.copy(), dt=configs.ROD_DT if case["cells"] == "rods" else DT)
    elif k == "tile":
        pos, r, gpos, gr = _tile_inputs(case, seed)
        side = case["cells"] * configs.BIN
        n, ng = r.numel(), gr.numel()
        work_pos, vel = pos.clone(), torch.empty_like(pos)
        ct = torch.full((max(n, ng, 1),), YEAST, dtype=torch.int32, device="cuda")
        dom = _Domain([configs.box_geometry(side, side)], n,
                      dict(x=work_pos[0], y=work_pos[1], z=work_pos[2], radius=r, cell_type=ct, velx=vel[0],
                           vely=vel[1], velz=vel[2]), {})
        t = abi.Tile()
        t.lo[:] = [0, 0, 0]
        t.hi[:] = [case["tile"] - 1, case["tile"] - 1, 31]
        S.update(dom=dom, ghosts=(gpos, gr, ct), start=pos, pos=work_pos, vel=vel, tile=t,
                 s_gh=_struct(ng, dict(x=gpos[0], y=gpos[1], z=gpos[2], radius=gr, cell_type=ct)))
    elif k == "host":
        pos, r = _spheres(case["n"], case["side"], seed)
        n = case["n"]

        def pinned(t):
            h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
            h.copy_(t)
            return h

        hp, hr = pinned(pos), pinned(r)
        ho = torch.empty((6, n), dtype=torch.float64, pin_memory=True)
        hc = pinned(torch.full((n,), YEAST, dtype=torch.int32))
        P = abi.Particles.__new__(abi.Particles)
        P.n, P.rods = n, False
        P.a = dict(x=hp[0].numpy(), y=hp[1].numpy(), z=hp[2].numpy(), radius=hr.numpy(), cell_type=hc.numpy())
        Q = abi.Particles.__new__(abi.Particles)
        Q.n, Q.rods, Q.a = n, False, {f: ho[i].numpy() for i, f in enumerate(SPHERE_OUT)}
        S.update(ctx=runtime.Context(configs.deck_params(), [configs.box_geometry(case["side"], case["side"])]),
                 P=P, Q=Q, out=ho, keep=(hp, hr, hc))
    elif k == "adjoint":
        n = case["n"]
        pos, r = _spheres(n, case["side"], seed)
        rng = np.random.default_rng(seed)
        out = torch.empty((6, n), dtype=torch.float64, device="cuda")
        inputs = dict(x=pos[0], y=pos[1], z=pos[2], radius=r,
                      cell_type=torch.full((n,), YEAST, dtype=torch.int32, device="cuda"))
        dom = _Domain([configs.box_geometry(case["side"], case["side"])], n, inputs, _planes(SPHERE_OUT[:3], out))
        S.update(dom=dom, out=out, adh=rng.uniform(0.0, 1.0e-3, n), grad=rng.normal(0.0, 1.0, (3, n)) / n)
    else:
        rec, mothers, draws = _split_records(case, seed)
        sp = abi.SplitParams(max_vol=5.0e-10, overlap=0.2, max_len=0.0035, max_rad=0.00025, brnch_prob=0.0,
                             split_prob=0.1, split_len=0.0030, num_reals=9, num_ints=0)
        S.update(rec=rec, mothers=mothers, kept=rec[mothers].clone(), draws=draws, sp=sp)
    return S


# ---- one pass ------------------------------------------------------------------

def run(S):
    case = S["case"]
    k = case["kind"]
    if k == "spheres":
        d = S["dom"]
        d.load()
        d.ctx.step(DT, case["steps"], PRECISION[case["precision"]])
        d.store()
        vel = S["out"][3:]
        if case["precision"] == "fp32f":
            with torch.cuda.stream(d.stream):
                vel = vel.float()
        return {"pos": S["out"][:3], "vel": vel}
    if k == "rods":
        d = S["dom"]
        d.load()
        d.ctx.step(configs.ROD_DT, case["steps"], PRECISION[case["precision"]])
        d.store()
        if case["precision"] == "fp64":
            return S["out"]
        with torch.cuda.stream(d.stream):
            return {f: t.float() if f in ("velx", "vely", "velz", "wx", "wy", "wz") else t
                    for f, t in S["out"].items()}
    if k == "aos":
        rec, ctx = S["rec"], S["ctx"]
        rec[...] = S["start"]
        cost = (C.c_double * 1)()
        nsub = C.c_int32(0)
        rc = ctx.lib.bmxg_evolve_particles_aos(ctx.h, rec.ctypes.data_as(C.c_void_p), len(rec), 34, 35, None, S["dt"],
                                               cost, C.byref(nsub))
        if rc:
            raise runtime.BmxgError(rc, ctx.lib.bmxg_last_error(ctx.h).decode())
        return {"pos": rec["pos"], "reals": rec["rdata"], "ints": rec["idata"]}
    if k == "tile":
        d = S["dom"]
        with torch.cuda.stream(d.stream):
            S["pos"].copy_(S["start"])
        d.check(d.ctx.lib.bmxg_step_tile(d.ctx.h, C.byref(S["tile"]), C.byref(d.s_in), C.byref(S["s_gh"]), DT,
                                         BMXG_DEVICE))
        return {"pos": S["pos"], "vel": S["vel"]}
    if k == "host":
        ctx = S["ctx"]
        ctx.set_state(S["P"], fields=SPHERE_IN)
        ctx.evolve_particles(DT)
        ctx.get_state(S["Q"], SPHERE_OUT)
        return {"pos": S["out"][:3], "vel": S["out"][3:]}
    if k == "adjoint":
        d = S["dom"]
        d.load()
        d.ctx.set_ext(0.05, 1.0e-2, S["adh"])
        d.ctx.forward(DT, case["steps"], case["every"])
        d.store()
        gx, gp, ga = d.ctx.backward(S["grad"])
        return {"pos": S["out"][:3], "grad_pos": gx, "grad_params": gp, "grad_adhesion": ga}
    rec, n = S["rec"], case["n"]
    rec[S["mothers"]] = S["kept"]
    m = runtime.split_cells_aos(rec.data_ptr(), n, S["sp"], draws=(S["draws"].data_ptr(), S["draws"].numel()),
                                next_id=n + 1, where=BMXG_DEVICE, cap=rec.shape[0])
    return {"reals": rec[:n + m, :37], "ints": rec.view(torch.int32)[:n + m, 74:111]}


# ---- the same in plain torch, 64 bits ---------------------------------------------

def _candidates(pos, colony, cells, side):
    """Ordered pairs (i, j, shift) of particles in adjacent bins, one block per
    bin offset: x and y periodic, z closed, bins of the level's cells."""
    nx, nz = cells
    lz = 0.064
    bx = torch.floor(pos[0] * (nx / side)).long().clamp(0, nx - 1)
    by = torch.floor(pos[1] * (nx / side)).long().clamp(0, nx - 1)
    bz = torch.floor(pos[2] * (nz / lz)).long().clamp(0, nz - 1)
    key = ((colony * nx + bx) * nx + by) * nz + bz
    skey, perm = torch.sort(key)
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                cx, cy, cz = bx + dx, by + dy, bz + dz
                ok = (cz >= 0) & (cz < nz)
                sx = torch.where(cx < 0, -1.0, 0.0) + torch.where(cx >= nx, 1.0, 0.0)
                sy = torch.where(cy < 0, -1.0, 0.0) + torch.where(cy >= nx, 1.0, 0.0)
                q = ((colony * nx + cx % nx) * nx + cy % nx) * nz + cz
                lo = torch.searchsorted(skey, q)
                num = torch.where(ok, torch.searchsorted(skey, q, right=True) - lo, torch.zeros_like(lo))
                i = torch.repeat_interleave(torch.arange(num.numel(), device=num.device), num)
                first = torch.cumsum(num, 0) - num
                j = perm[lo[i] + torch.arange(i.numel(), device=num.device) - first[i]]
                keep = i != j
                i, j = i[keep], j[keep]
                yield i, j, sx[i].double() * side, sy[i].double() * side


def _wall(z, rS, P):
    dz = z - P.z_wall
    rA = rS + P.z_bndry_width
    near = -P.z_stiffness * (dz - rA) ** 2 * (dz - rS)
    v = torch.where(dz <= 0, P.z_stiffness * rA * rA * rS, torch.where(dz < rA, near, torch.zeros_like(dz)))
    return v - P.z_gravity * P.z_stiffness * rA * rA * rS


def _close_pairs(pos, r, colony, cells, side, P):
    out = []
    for i, j, sx, sy in _candidates(pos, colony, cells, side):
        d0 = pos[0][i] - (pos[0][j] + sx)
        d1 = pos[1][i] - (pos[1][j] + sy)
        d2 = pos[2][i] - pos[2][j]
        near = d0 * d0 + d1 * d1 + d2 * d2 < (r[i] + r[j] + P.bndry_width) ** 2
        out.append((i[near], j[near], sx[near], sy[near]))
    return [torch.cat(c) for c in zip(*out)]


def _sphere_velocity(pos, r, pairs, P, gamma=None, mu=0.0, adh=None, k=None):
    i, j, sx, sy = pairs
    k = P.stiffness if k is None else k
    d = torch.stack([pos[0][i] - (pos[0][j] + sx), pos[1][i] - (pos[1][j] + sy), pos[2][i] - pos[2][j]])
    dist = d.square().sum(0).sqrt()
    rS = r[i] + r[j]
    e = dist - (rS + P.bndry_width)
    F = -k * e * e * (dist - rS)
    v = torch.zeros_like(pos)
    if gamma is not None:
        m = 1.0 / (6.0 * math.pi * mu * r)
        F = F - k * P.bndry_width * 0.5 * (adh[i] + adh[j]) * e * e
        F = F / (1.0 + gamma * (m[i] + m[j]))
        v = v.index_add(1, i, F * d / dist) * m
    else:
        v = v.index_add(1, i, F * d / dist)
    return v + torch.stack([torch.zeros_like(pos[2]), torch.zeros_like(pos[2]), _wall(pos[2], r, P)])


def _wrap(pos, side):
    return torch.stack([pos[0] - side * torch.floor(pos[0] / side), pos[1] - side * torch.floor(pos[1] / side),
                        pos[2]])


def _exact_spheres(pos, r, colony, side, steps):
    P = configs.deck_params()
    cells = (int(round(side / configs.BIN)), 32)
    vel = torch.zeros_like(pos)
    for _ in range(steps):
        vel = _sphere_velocity(pos, r, _close_pairs(pos, r, colony, cells, side, P), P)
        pos = _wrap(pos + DT * vel, side)
    return pos, vel


def _seg_closest(a1, u, b1, v):
    """Parameters of the closest points of segments a1 + s u and b1 + t v, s and
    t in [0, 1] (3 x m each): the unconstrained solution where it lies inside,
    else the best of the four edges' clamped minima."""
    w = a1 - b1
    a, b, c = (u * u).sum(0), (u * v).sum(0), (v * v).sum(0)
    d, e = (u * w).sum(0), (v * w).sum(0)
    det = a * c - b * b
    s0, t0 = (b * e - c * d) / det, (a * e - b * d) / det
    cand = [(torch.zeros_like(a), (e / c).clamp(0, 1)), (torch.ones_like(a), ((e + b) / c).clamp(0, 1)),
            ((-d / a).clamp(0, 1), torch.zeros_like(a)), (((b - d) / a).clamp(0, 1), torch.ones_like(a))]
    s, t = cand[0]
    best = (w + s * u - t * v).square().sum(0)
    for cs, ct in cand[1:]:
        q = (w + cs * u - ct * v).square().sum(0)
        s, t, best = torch.where(q < best, cs, s), torch.where(q < best, ct, t), torch.minimum(q, best)
    inside = (s0 >= 0) & (s0 <= 1) & (t0 >= 0) & (t0 <= 1) & (det > 0)
    return torch.where(inside, s0, s), torch.where(inside, t0, t)


def _exact_rods(T, side, steps):
    """The segments' step: bonded springs, closest-point contact, mobility, the
    growth surface on both ends, translation and rotation of the axis."""
    P = configs.deck_params()
    cells = (int(round(side / configs.BIN)), 32)
    pos, th, ph = T["pos"], T["theta"], T["phi"]
    L, rad, n = T["c_length"], T["radius"], T["c_length"].numel()
    colony = torch.zeros(n, dtype=torch.long, device=pos.device)
    ids, site, nb = T["seg_id1"].reshape(4, n), T["site"].reshape(4, n), T["n_bnds"]
    arad = torch.sqrt(T["area"] / 2.0 / (4.0 * math.pi))
    d0 = 1.0 / (6.0 * math.pi * arad * P.viscosity)
    da = (L * L - 2.0 * arad * arad / 3.0) / (4.0 * math.pi * L ** 3 * P.viscosity)
    db = (L * L + 2.0 * arad * arad / 3.0) / (8.0 * math.pi * L ** 3 * P.viscosity)
    vel = rot = torch.zeros_like(pos)
    for _ in range(steps):
        ct, st, cp, sp = torch.cos(th), torch.sin(th), torch.cos(ph), torch.sin(ph)
        ax = torch.stack([st * cp, st * sp, ct])
        Sv, Dv = torch.zeros_like(pos), torch.zeros_like(pos)
        for i, j, sx, sy in _candidates(pos, colony, cells, side):
            d = torch.stack([pos[0][i] - (pos[0][j] + sx), pos[1][i] - (pos[1][j] + sy), pos[2][i] - pos[2][j]])
            keep = d.square().sum(0) <= (1.5 * (L[i] + L[j]) + P.bndry_width - 1.0e-15) ** 2
            i, j, d = i[keep], j[keep], d[:, keep]
            u, v = ax[:, i] * L[i], ax[:, j] * L[j]
            a1, b1 = d - 0.5 * u, -0.5 * v
            si, sj = torch.zeros_like(i), torch.zeros_like(i)
            for m in (3, 2, 1, 0):
                si = torch.where((nb[i] > m) & (ids[m][i] == j + 1), site[m][i].long(), si)
                sj = torch.where((nb[j] > m) & (ids[m][j] == i + 1), site[m][j].long(), sj)
            bonded = (si > 0) & (sj > 0)
            s, t = _seg_closest(a1, u, b1, v)
            g = (a1 + s * u) - (b1 + t * v)
            dist = g.square().sum(0).sqrt()
            rS = rad[i] + rad[j]
            e = dist - (rS + P.bndry_width)
            F = torch.where(e < 0, -P.stiffness * e * e * (dist - rS), torch.zeros_like(e))
            F = F * g / torch.where(dist > 1.0e-8, dist, torch.ones_like(dist))
            spring = -P.bond_strength * ((a1 + torch.where(si == 2, 1.0, 0.0) * u) -
                                         (b1 + torch.where(sj == 2, 1.0, 0.0) * v))
            f1 = torch.where(bonded, torch.where(si == 1, spring, torch.zeros_like(F)), F * (1.0 - s))
            f2 = torch.where(bonded, torch.where(si == 2, spring, torch.zeros_like(F)), F * s)
            Sv.index_add_(1, i, f1 + f2)
            Dv.index_add_(1, i, f1 - f2)
        rv = -ax * L
        vel = 0.5 * ((d0 + db) * Sv + (da - db) * (ax * Sv).sum(0) * ax)
        rot = 0.5 * (d0 - db) * torch.linalg.cross(rv, Dv, dim=0)
        zero = torch.zeros_like(ct)
        w1 = torch.stack([zero, zero, _wall(pos[2] - 0.5 * ct * L, rad, P)])
        w2 = torch.stack([zero, zero, _wall(pos[2] + 0.5 * ct * L, rad, P)])
        un = rv / rv.square().sum(0).sqrt()
        fn = ((w1 - w2) * un).sum(0)
        w1, w2 = w1 - 0.5 * fn * un, w2 + 0.5 * fn * un
        vw = 0.5 * (w1 + w2)
        vel = vel + vw
        rot = rot + 0.5 * torch.linalg.cross(rv, w1 - w2, dim=0)
        # the axis turned by |omega| dt about the rotation's part across it
        o1 = (-sp * rot[0] + cp * rot[1]) * 2.0 / (L * L)
        o2 = (-cp * ct * rot[0] - sp * ct * rot[1] + st * rot[2]) * 2.0 / (L * L)
        on = torch.sqrt(o1 * o1 + o2 * o2)
        ang = on * configs.ROD_DT
        den = torch.where(on > 0, on, torch.ones_like(on))
        q0, q1, q2 = torch.cos(ang), o2 / den * torch.sin(ang), -o1 / den * torch.sin(ang)
        nd = torch.stack([cp * st * q0 - sp * q1 - cp * ct * q2, sp * st * q0 + cp * q1 - sp * ct * q2,
                          ct * q0 + st * q2])
        th = torch.acos(nd[2])
        rho = torch.sqrt(nd[0] ** 2 + nd[1] ** 2)
        ph = torch.acos((nd[0] / rho).clamp(-1.0, 1.0))
        ph = torch.where(nd[1] < 0, 2.0 * math.pi - ph, ph)
        pos = _wrap(pos + configs.ROD_DT * vel, side)
    return pos, th, ph, vel, rot


def _rod_tensors(P):
    T = {f: torch.from_numpy(np.ascontiguousarray(P[f])).cuda()
         for f in ("theta", "phi", "c_length", "radius", "area", "n_bnds", "seg_id1", "site")}
    T["pos"] = torch.from_numpy(np.stack([P["x"], P["y"], P["z"]])).cuda()
    return T


def exact(case, seed):
    k = case["kind"]
    if k == "spheres":
        off = _colony_order(case, seed)
        n = int(off[-1])
        if n * case["steps"] > 300_000_000:
            return None
        pos, r = _spheres(n, case["side"], seed)
        colony = torch.repeat_interleave(torch.arange(len(off) - 1, device="cuda"),
                                         torch.from_numpy(np.diff(off)).cuda())
        pos, vel = _exact_spheres(pos, r, colony, case["side"], case["steps"])
        return {"pos": pos, "vel": vel.float() if case["precision"] == "fp32f" else vel}
    if k == "rods":
        T = _rod_tensors(_trees(case["trees"], case["per_tree"], case["side"], seed))
        pos, th, ph, vel, rot = _exact_rods(T, case["side"], case["steps"])
        if case["precision"] == "fp32f":
            vel, rot = vel.float(), rot.float()
        out = dict.fromkeys(ROD_OUT)
        out.update(x=pos[0], y=pos[1], z=pos[2], theta=th, phi=ph, velx=vel[0], vely=vel[1], velz=vel[2], wx=rot[0],
                   wy=rot[1], wz=rot[2])
        return out
    if k == "aos":
        P = _aos_particles(case, seed)
        rec = _records(P)
        R = abi.REAL_IDX
        if case["cells"] == "rods":
            pos, th, ph, vel, rot = _exact_rods(_rod_tensors(P), _aos_side(case), 1)
            rec["rdata"][:, R["theta"]], rec["rdata"][:, R["phi"]] = th.cpu().numpy(), ph.cpu().numpy()
            rec["rdata"][:, R["wx"]:R["wz"] + 1] = rot.T.cpu().numpy()
        else:
            p = torch.from_numpy(np.stack([P["x"], P["y"], P["z"]])).cuda()
            r = torch.from_numpy(P["radius"]).cuda()
            pos, vel = _exact_spheres(p, r, torch.zeros(P.n, dtype=torch.long, device="cuda"), case["side"], 1)
        rec["rdata"][:, R["velx"]:R["velz"] + 1] = vel.T.cpu().numpy()
        return {"pos": pos.T.contiguous().cpu().numpy(), "reals": rec["rdata"], "ints": None}
    if k == "tile":
        pos, r, gpos, gr = _tile_inputs(case, seed)
        P = configs.deck_params()
        side = case["cells"] * configs.BIN
        n = r.numel()
        # a box wide enough that the copies are far from its faces: no images
        allp = torch.cat([pos, gpos], dim=1)
        allp[:2] += side
        allr = torch.cat([r, gr])
        zero = torch.zeros(allr.numel(), dtype=torch.long, device="cuda")
        pairs = _close_pairs(allp, allr, zero, (3 * case["cells"], 32), 3.0 * side, P)
        mine = pairs[0] < n
        allp[:2] -= side
        vel = _sphere_velocity(allp, allr, [c[mine] for c in pairs], P)[:, :n]
        return {"pos": _wrap(pos + DT * vel, side), "vel": vel}
    if k == "host":
        pos, r = _spheres(case["n"], case["side"], seed)
        zero = torch.zeros(case["n"], dtype=torch.long, device="cuda")
        pos, vel = _exact_spheres(pos, r, zero, case["side"], 1)
        return {"pos": pos, "vel": vel}
    if k == "adjoint":
        P = configs.deck_params()
        n, side = case["n"], case["side"]
        x0, r = _spheres(n, side, seed)
        rng = np.random.default_rng(seed)
        adh = torch.from_numpy(rng.uniform(0.0, 1.0e-3, n)).cuda().requires_grad_()
        g = torch.from_numpy(rng.normal(0.0, 1.0, (3, n)) / n).cuda()
        par = [torch.tensor(v, dtype=torch.float64, device="cuda", requires_grad=True)
               for v in (P.stiffness, 0.05, 1.0e-2)]
        x0.requires_grad_()
        pos = x0
        cells = (int(round(side / configs.BIN)), 32)
        zero = torch.zeros(n, dtype=torch.long, device="cuda")
        for _ in range(case["steps"]):
            with torch.no_grad():
                pairs = _close_pairs(pos, r, zero, cells, side, P)
            vel = _sphere_velocity(pos, r, pairs, P, gamma=par[1], mu=par[2], adh=adh, k=par[0])
            pos = pos + DT * vel
            pos = pos - torch.stack([side * torch.floor(pos[0].detach() / side),
                                     side * torch.floor(pos[1].detach() / side), torch.zeros_like(pos[2])])
        grads = torch.autograd.grad((pos * g).sum(), [x0, adh] + par)
        return {"pos": pos.detach(), "grad_pos": grads[0], "grad_params": torch.stack(grads[2:]),
                "grad_adhesion": grads[1]}
    rec, mothers, draws = _split_records(case, seed)
    n, m = case["n"], mothers.numel()
    R = abi.REAL_IDX
    reals = rec[:n + m, :37].clone()
    old = reals[mothers]
    u = draws[:2 * m].reshape(m, 2)
    th, ph = torch.acos(2.0 * u[:, 0] - 1.0), 2.0 * math.pi * u[:, 1]
    axis = torch.stack([torch.sin(th) * torch.cos(ph), torch.sin(th) * torch.sin(ph), torch.cos(th)], dim=1)
    step = 0.8 * 0.5 * axis * old[:, 3 + R["radius"], None]
    vol = old[:, 3 + R["vol"]] / 2.0
    radius = (3.0 * vol / (4.0 * math.pi)) ** (1.0 / 3.0)
    new = old.clone()
    new[:, 3 + R["vol"]] = vol
    new[:, 3 + R["radius"]] = radius
    new[:, 3 + R["area"]] = 4.0 * math.pi * radius * radius
    new[:, 3 + R["dadt"]] = 2.0 * old[:, 3 + R["dvdt"]] / radius
    new[:, 3 + 31:3 + 34] *= 0.5
    kid = new.clone()
    new[:, :3] = old[:, :3] - step
    kid[:, :3] = old[:, :3] + step
    kid[:, 3 + R["bond_scale"]] = 1.0
    reals[mothers] = new
    reals[n:] = kid
    return {"reals": reals, "ints": None}
