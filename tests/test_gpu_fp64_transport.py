"""The FP64 transport (k_transport_radial_march, k_transport_azimuthal_warp) against the
oracle's, at the sizes where its split can go wrong: rings of less, exactly and more
than a warp's and a block's sectors (30 and 31, 120, 124, 960), grids of fewer rings than a chunk's
lead, the wrap of the last sector, rows that are not 16-byte strided, and densities
for which rho / (rho + 1e-20) is not 1, down to empty cells.

Tolerance: limited slopes are formed within 2^-43 and enter a cell once per sweep with a
Courant factor below 1, times differences of at most twice the field's maximum, in three
sweeps: 6 x 2^-43 = 7e-13 of the maximum, plus some 60 roundings (7e-15).  A velocity
is a momentum over a density, of contrast at most 3 where it is compared.
"""
import numpy as np
import pytest

import cudaprotoplanetarydisks_gb300 as fg
from oracle.oracle import OracleDisk
from tests.helpers import rel_linf, small

pytestmark = pytest.mark.gpu
TOL = 1e-12

SHAPES = [(8, 30), (9, 31), (15, 32), (16, 61), (33, 62), (8, 120), (9, 123), (65, 124), (12, 125), (40, 249), (8, 961), (8, 1000)]


def fields(params, low, seed):
    rng = np.random.default_rng(seed)
    n, m = params.nrad + 1, params.nsec
    f = dict(dens=params.sigma0 * rng.uniform(0.5, 1.5, (n, m)), vrad=0.02 * rng.normal(size=(n, m)),
             vtheta=1.0 + 0.02 * rng.normal(size=(n, m)), energy=params.sigma0 * 1e-3 * rng.uniform(0.5, 1.5, (n, m)))
    if low:  # a third of the cells between 1e-24 and 1e-4, some empty
        pick = rng.random((n, m)) < 1 / 3
        f["dens"][pick] = 10 ** rng.uniform(-24, -4, pick.sum())
        f["dens"][rng.random((n, m)) < 0.02] = 0.0
    for v in f.values():
        v[-1] = 0.0
    f["vrad"][0] = 0.0
    return f


def run(d, f, dt):
    d.set_fields(f["dens"], f["vrad"], f["vtheta"], f["energy"])
    d.substep(fg.SUB_TRANSPORT, dt)
    return {k: d.field(k) for k in f}


@pytest.mark.parametrize("low", [False, True])
@pytest.mark.parametrize("cfg", ["c1", "c3"])
@pytest.mark.parametrize("nrad,nsec", SHAPES)
def test_fp64_transport(cfg, nrad, nsec, low):
    params, planets = small(cfg, nrad=nrad, nsec=nsec)
    # a Courant factor below 1/2 for the fastest of the random velocities
    dt = 0.25 * min((params.rmax / params.rmin) ** (1 / nrad) - 1, 2 * np.pi / nsec) * params.rmin / 0.1
    f = fields(params, low, nrad * 1000 + nsec)
    ref = OracleDisk(params, planets)
    want = run(ref, f, dt)
    got = []
    for v in (dict(), dict(rad_tma=0), dict(rad_col=1)):
        var = fg.default_variant()
        for k, x in v.items():
            setattr(var, k, x)
        b = fg.Batch([(params, planets)], fg.FARGO_FP64, variant=var)
        got.append(run(b.disk(0), f, dt))
        b.close()
    names = ["dens"] + (["energy"] if cfg == "c3" else []) + ([] if low else ["vrad", "vtheta"])
    for k in names:
        assert np.isfinite(got[0][k]).all(), k
        assert rel_linf(got[0][k], want[k]) < TOL * (3 if k[0] == "v" else 1), k
    for other in got[1:]:
        for k in f:
            assert np.array_equal(other[k][:-1], got[0][k][:-1], equal_nan=True), k
