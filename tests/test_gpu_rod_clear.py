"""The FP32 range screen of rod contacts (rod_clear32: a pair certainly out of
contact range adds exact zeros and is not queued) against the oracle, which
evaluates every gated pair: short and long segments, thick and thin, random,
axis-aligned, exactly parallel and nearly perpendicular axes, crossing, touching
and just out of range, in both forms."""
import numpy as np
import pytest

from boltzmannmfx_gb300 import Context, abi, configs
from boltzmannmfx_gb300.abi import BMXG_FP32F, BMXG_FP64, FUNGI
from oracle import oracle as O

from common import trig_floor, within

pytestmark = pytest.mark.gpu


def segments(n, angles, lmax, rmax, seed):
    rng = np.random.default_rng(seed)
    P = abi.Particles(n, rods=True)
    side = 0.016
    P["x"], P["y"] = rng.uniform(0, side, n), rng.uniform(0, side, n)
    P["z"] = rng.uniform(0.044, 0.050, n)
    if angles == "random":
        P["theta"], P["phi"] = np.arccos(rng.uniform(-1, 1, n)), rng.uniform(0, 2 * np.pi, n)
    elif angles == "axes":
        P["theta"] = rng.choice([0.0, np.pi / 2, np.pi], n)
        P["phi"] = rng.choice([0.0, np.pi / 2, np.pi, 1.5 * np.pi], n)
    else:
        P["theta"], P["phi"] = 1.1, 0.3
    if angles == "nearly":
        P["theta"] += rng.normal(0.0, 1.0e-6, n)
        P["phi"] += rng.choice([0.0, np.pi / 2], n) + rng.normal(0.0, 3.0e-5, n)
    P["c_length"] = np.exp(rng.uniform(np.log(lmax / 30), np.log(lmax), n))
    P["radius"] = rng.uniform(rmax / 10, rmax, n)
    P["area"] = 2 * np.pi * P["radius"] * (P["c_length"] + P["radius"])
    P["cell_type"] = FUNGI
    P["position"] = abi.SITE_INTERIOR
    return configs.deck_params(), configs.box_geometry(side, side), P


@pytest.mark.parametrize("angles", ["random", "axes", "parallel", "nearly"])
@pytest.mark.parametrize("n, lmax, rmax", [(400, 0.004, 2.0e-4), (300, 0.012, 6.0e-4), (500, 0.0005, 4.0e-4)])
def test_screened_contacts_equal_the_oracle(gpu_lib, angles, n, lmax, rmax):
    prm, g, P = segments(n, angles, lmax, rmax, n)
    pl = O.pairs(prm, g, P)
    fc = O.forces(prm, g, P.copy(), pl)
    fv, fw = trig_floor(O, prm, g, P)
    for prec, rel in ((BMXG_FP64, 1.0e-10), (BMXG_FP32F, 1.0e-5)):
        ctx = Context(prm, [g])
        ctx.set_state(P)
        ctx.step(configs.ROD_DT, 1, prec)
        Q = P.copy()
        ctx.get_state(Q)
        ctx.close()
        got = np.stack([Q[k] for k in ("velx", "vely", "velz", "wx", "wy", "wz")])
        assert within(got[:3], fc[:3], rel, 8 * fv)
        assert within(got[3:], fc[3:], rel, 8 * fw)
