"""The FP32 source step's divides at the ends of the exponent range: they are IEEE quotients, in the
kernels with one thread per cell and in the march that a batch of a million cells takes (k_gas).

Without an energy equation and a planet the source step only has densities in quotients of the
same degree, so a density times a power of two leaves the velocities as they are, bit for
bit, as long as nothing is subnormal.  Far out the artificial viscosity has subnormals (its pressure
below, its factor 2 dt / (rho + rho') above): at most 2^-150 of at most 2^116 over a cell of 2^-7, which
leaves the velocities, of about 1, within two ulps.
"""
import numpy as np
import pytest

import cudaprotoplanetarydisks_gb300 as fg
from tests.helpers import small

pytestmark = pytest.mark.gpu
NRAD, NSEC, DT = 24, 130, 2e-3


def fields(rng, scale=1.0):
    shape = (NRAD + 1, NSEC)
    # 8 bits, within 5% of 2^-10.6
    dens = 2.0 ** -11 * rng.integers(332, 350, shape) / 256.0 * scale
    f = dict(dens=dens, vrad=0.02 * rng.normal(size=shape), vtheta=1.0 + 0.02 * rng.normal(size=shape))
    for v in f.values():
        v[-1] = 0.0
    f["vrad"][0] = 0.0
    return f


def disks(cfg="c1", **kw):
    """The same disk alone (cell kernels) and beside a million cells (k_gas)."""
    params, _ = small(cfg, nrad=NRAD, nsec=NSEC, sigmaslope=0.0, **kw)
    batch = fg.Batch([(params, []), small("c1", nrad=1000, nsec=1000)], fg.FARGO_FP32_BULK)
    return params, fg.Disk(params, [], fg.FARGO_FP32_BULK), batch


def source(d, f, *parts):
    d.set_fields(**f)
    for which in (fg.SUB_SOURCE, *parts):
        d.substep(which, DT)
    return {k: d.field(k) for k in f}


@pytest.mark.parametrize("power,ulps", [(-60, 0), (60, 0), (100, 0), (-100, 2), (136, 2)])
def test_source_step_of_scaled_densities(power, ulps):
    params, alone, batch = disks()
    for d in (alone, batch.disk(0)):
        want = source(d, fields(np.random.default_rng(5)))
        got = source(d, fields(np.random.default_rng(5), 2.0 ** power))
        for k in ("vrad", "vtheta"):
            assert np.abs(got[k] - want[k])[:-1].max() <= ulps * 2.0 ** -23, k
    batch.close()


def test_source_step_of_subnormal_densities():
    params, alone, batch = disks()
    f = fields(np.random.default_rng(6), 2.0 ** -117)  # sums of two: about 2^-126.6
    wide = fg.Disk(params, [], fg.FARGO_FP64)
    want = source(wide, f)
    rinf = wide.mesh()[0]
    # a pressure (about 2^-136) is a subnormal, off by 2^-149 at most after its two products; over a sum of
    # at least 2^-127, times 2 for the difference and 2 for the formula's factor, over the narrowest cell
    tol = DT * 2.0 ** -20 / min(np.diff(rinf).min(), rinf[0] * 2 * np.pi / NSEC) + 1e-6
    for d in (alone, batch.disk(0)):
        got = source(d, f)
        for k in ("vrad", "vtheta"):
            assert np.abs(got[k] - want[k])[:-1].max() < tol, k
    batch.close()


@pytest.mark.parametrize("cfg", ["c1", "c3"])
def test_gas_march_is_bitwise_the_cell_kernels_at_the_ends_of_the_range(cfg):
    params, alone, batch = disks(cfg)
    rng = np.random.default_rng(7)
    f = fields(rng)
    odd = [0.0, 1e-45, 3e-39, 1.2e-38, 1e-30, 1e30, 8.6e37, 1.7e38, 3e38, np.inf, np.nan, -1e-3]
    for n, v in enumerate(odd):  # well apart: each meets ordinary neighbours
        f["dens"][2 * n % 20 + 1, 10 * n + 3] = v
    f["dens"][:, :2] = 0.0
    f["dens"][:, 2] = 2e-39
    if cfg == "c3":
        f["energy"] = 1e-3 * params.sigma0 * rng.uniform(0.5, 1.5, f["dens"].shape)
        f["energy"][4, 5::7] = 3e38
        f["energy"][9, 5::7] = 1e-42
    parts = (fg.SUB_ENERGY,) if cfg == "c3" else ()
    a, b = source(alone, f, *parts), source(batch.disk(0), f, *parts)
    for k in a:
        assert np.array_equal(a[k], b[k], equal_nan=True), k
    assert np.isfinite(a["vrad"]).mean() > 0.5
    batch.close()
