"""The FP64 source step and energy equation (source_cell, visc_tau_cell, visc_update_body,
artvisc_body, energy_body in their FP64 forms) against the oracle's, on rings that are
no multiple of a warp or a block, with and without a planet's potential, with self-gravity, with a
rotating frame, with and without cooling.

Tolerance: a velocity takes some 60 roundings of terms of at most a few times its
largest value (v up to about 1 on rings whose spacing keeps dt v / dr below 1): 60 x 2^-53 x 10 =
7e-14, 1e-13 here; divergence and Q+ come from differences of 2% of the velocities: 50 times that.
"""
import numpy as np
import pytest

import cudaprotoplanetarydisks_gb300 as fg
from oracle.oracle import OracleDisk
from tests.helpers import rel_linf, small

pytestmark = pytest.mark.gpu

CASES = [("c1", 8, 9, {}), ("c1", 33, 65, {}), ("c1", 12, 260, dict(nb=0)), ("c2", 16, 48, {}), ("c2", 24, 96, dict(adiabatic=1)),
         ("c3", 9, 31, {}), ("c3", 21, 130, {}), ("c3", 17, 67, dict(cooling=0)), ("c3", 16, 64, dict(nb=0)),
         ("c3", 40, 129, dict(corotating=1)), ("c1", 10, 33, dict(imposeddiskdrift=1e-3))]


@pytest.mark.parametrize("cfg,nrad,nsec,extra", CASES)
def test_fp64_source_and_energy(cfg, nrad, nsec, extra):
    params, planets = small(cfg, nrad=nrad, nsec=nsec, **{k: v for k, v in extra.items() if k != "nb"})
    if "nb" in extra:
        planets = []
    rng = np.random.default_rng(nrad * 1000 + nsec)
    disk, ref = fg.Disk(params, planets, fg.FARGO_FP64), OracleDisk(params, planets)
    f = {k: ref.field(k) for k in ("dens", "vrad", "vtheta", "energy")}
    shape = f["dens"].shape
    for k in ("dens", "energy"):
        f[k] *= rng.uniform(0.8, 1.2, shape)
    f["vtheta"] += 0.02 * rng.normal(size=shape)
    f["vrad"] += 0.02 * rng.normal(size=shape)
    f["vrad"][0] = 0.0
    for v in f.values():
        v[-1] = 0.0
    dt = 1e-3
    for d in (disk, ref):
        d.set_fields(f["dens"], f["vrad"], f["vtheta"], f["energy"])
        d.substep(fg.SUB_POTENTIAL, dt)
        d.substep(fg.SUB_SOURCE, dt)
    names = ["vrad", "vtheta", "pressure"]
    for k in names:
        assert rel_linf(disk.field(k), ref.field(k)) < 1e-13, k
    if params.adiabatic:
        for d in (disk, ref):
            d.substep(fg.SUB_ENERGY, dt)
        assert rel_linf(disk.field("energy"), ref.field("energy")) < 1e-13
        for k in ("divergence", "qplus"):
            assert rel_linf(disk.field(k), ref.field(k)) < 5e-12, k
