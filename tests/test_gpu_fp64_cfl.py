"""The FP64 CFL/force kernel at the sizes of both its forms (four cells per thread for
260 <= nsec <= 1024 and nsec % 4 == 0, streamed otherwise) against the oracle: the time-step
limit, whose largest cell FP32 estimates pick out, on random, axisymmetric (every cell of a
ring ties) and cold disks (the estimates' differences cancel), the planets' potential and the
disk's pull on the planets.

ConditionCFL returns ceil(deltaT / limit): equal integers up to 1e7 fix the limit to 1e-7.
Potential: 1/d within 2 roundings, the distance's own rounding magnified at the planet by
distance / smoothing (at most 60): 60 x 2^-52 of the largest, twice (both sides) = 3e-14.
"""
import numpy as np
import pytest

import cudaprotoplanetarydisks_gb300 as fg
from oracle.oracle import OracleDisk
from tests.helpers import rel_linf, small

pytestmark = pytest.mark.gpu


def pair(cfg, nrad, nsec, kind):
    extra = dict(aspectratio=1e-3) if kind == "cold" else {}
    params, planets = small(cfg, nrad=nrad, nsec=nsec, **extra)
    disk, ref = fg.Disk(params, planets, fg.FARGO_FP64), OracleDisk(params, planets)
    rng = np.random.default_rng(nrad * 10000 + nsec)
    f = {k: ref.field(k) for k in ("dens", "vrad", "vtheta", "energy")}
    shape = f["dens"].shape
    if kind == "axisymmetric":
        for k in f:
            f[k][:] = f[k][:, :1]
    else:
        f["dens"] *= rng.uniform(0.5, 1.5, shape)
        f["vrad"] += (1e-6 if kind == "cold" else 0.05) * rng.normal(size=shape)
        f["vtheta"] += (1e-6 if kind == "cold" else 0.05) * rng.normal(size=shape)
    f["vrad"][0] = 0.0
    for v in f.values():
        v[-1] = 0.0
    for d in (disk, ref):
        d.set_fields(f["dens"], f["vrad"], f["vtheta"], f["energy"])
    return disk, ref


@pytest.mark.parametrize("kind", ["random", "axisymmetric", "cold"])
@pytest.mark.parametrize("cfg,nrad,nsec", [("c1", 8, 9), ("c3", 16, 67), ("c1", 20, 256), ("c3", 11, 260), ("c1", 24, 384),
                                           ("c1", 9, 1024), ("c3", 8, 1028), ("c2", 16, 96), ("c2", 16, 288)])
def test_fp64_cfl_and_potential(cfg, nrad, nsec, kind):
    disk, ref = pair(cfg, nrad, nsec, kind)
    for deltaT in (1e-4, 0.05, 0.314159265359, 7.0, 1234.5, 3e4):
        n = ref.condition_cfl(deltaT)
        if n < 10 ** 7:
            assert disk.condition_cfl(deltaT) == n, deltaT
    for d in (disk, ref):
        d.substep(fg.SUB_POTENTIAL, 0.01)
    assert rel_linf(disk.field("potential"), ref.field("potential")) < 3e-14


@pytest.mark.parametrize("nrad,nsec", [(16, 96), (16, 288)])
def test_fp64_pull_on_planets(nrad, nsec):
    disk, ref = pair("c2", nrad, nsec, "random")
    for d in (disk, ref):
        d.substep_full(1e-3)
    for a, b in zip(disk.planets(), ref.planets()):
        for k in ("x", "y", "vx", "vy"):
            assert abs(getattr(a, k) - getattr(b, k)) < 1e-14, k
