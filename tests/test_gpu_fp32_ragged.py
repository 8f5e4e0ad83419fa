"""The FP32 azimuthal transport of rings that are no multiple of four sectors
(k_transport_azimuthal_warp32) against the kernel with a barrier per phase that it replaces there
(variant az_generic), on one transport step: rings of less, exactly and more than a warp's 120
sectors and a block's, wrapped shifts, densities down to empty cells, with and without
k_gas's separate fields.

Both round alike; only the ring mean's summation order differs (44 against 53 bits), which
moves a residual velocity by an ulp in rare cells: 4 ulps (2.4e-7) of each field's maximum.
"""
import numpy as np
import pytest

import cudaprotoplanetarydisks_gb300 as fg
from tests.helpers import rel_linf, small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("low", [False, True])
@pytest.mark.parametrize("cfg,nrad,nsec", [("c1", 8, 9), ("c3", 9, 30), ("c3", 12, 31), ("c1", 16, 119), ("c3", 8, 121), ("c1", 10, 122),
                                           ("c3", 17, 239), ("c1", 8, 241), ("c3", 8, 961), ("c1", 9, 1443)])
def test_fp32_ragged_rings(cfg, nrad, nsec, low):
    params, planets = small(cfg, nrad=nrad, nsec=nsec)
    rng = np.random.default_rng(nsec)
    shape = (nrad + 1, nsec)
    f = dict(dens=params.sigma0 * rng.uniform(0.5, 1.5, shape), vrad=0.02 * rng.normal(size=shape),
             vtheta=1.0 + 0.02 * rng.normal(size=shape), energy=params.sigma0 * 1e-3 * rng.uniform(0.5, 1.5, shape))
    if low:
        pick = rng.random(shape) < 1 / 3
        f["dens"][pick] = 10 ** rng.uniform(-24, -4, pick.sum())
        f["dens"][rng.random(shape) < 0.02] = 0.0
    for v in f.values():
        v[-1] = 0.0
    f["vrad"][0] = 0.0
    dt = 0.25 * min((params.rmax / params.rmin) ** (1 / nrad) - 1, 2 * np.pi / nsec) * params.rmin / 0.1

    def run(generic, beside):
        v = fg.default_variant()
        v.az_generic = generic
        b = fg.Batch([(params, planets)] + beside, fg.FARGO_FP32_BULK, variant=v)
        d = b.disk(0)
        d.set_fields(f["dens"], f["vrad"], f["vtheta"], f["energy"])
        d.substep(fg.SUB_TRANSPORT, dt)
        got = {k: d.field(k) for k in f}
        b.close()
        return got

    want = run(1, [])
    alone, gas = run(0, []), run(0, [small("c1", nrad=1000, nsec=1000)])
    names = ["dens"] + (["energy"] if cfg == "c3" else []) + ([] if low else ["vrad", "vtheta"])
    for k in names:
        assert np.isfinite(alone[k]).all(), k
        assert rel_linf(alone[k], want[k]) <= 2.4e-7, k
    for k in f:
        assert np.array_equal(alone[k], gas[k], equal_nan=True), k
