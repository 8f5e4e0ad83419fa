"""The residual velocities of the FP32 azimuthal transport on rings that are no multiple of four sectors
(k_transport_azimuthal_warp32) against the kernel with a barrier per phase (variant az_generic), which
forms Vtheta - mean (+ the constant residual, without the FARGO split) in FP64 and rounds
once.  Fields whose azimuthal velocities differ from the mean by more than a factor of two, with and without the split: the
two kernels' densities are equal but where their ring means (44 against 53 bits) round a residual differently,
less than one cell in a hundred.
"""
import numpy as np
import pytest

import cudaprotoplanetarydisks_gb300 as fg
from tests.helpers import small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fast", [0, 1])
@pytest.mark.parametrize("nrad,nsec", [(12, 241), (16, 1003)])
def test_residual_velocities(nrad, nsec, fast):
    params, planets = small("c1", nrad=nrad, nsec=nsec, fast_transport=fast)
    rng = np.random.default_rng(nsec)
    shape = (nrad + 1, nsec)
    f = dict(dens=params.sigma0 * rng.uniform(0.5, 1.5, shape), vrad=np.zeros(shape), vtheta=rng.uniform(0.0, 1.0, shape))
    for v in f.values():
        v[-1] = 0.0
    dt = 0.25 * 2 * np.pi / nsec * params.rmin / 1.0
    got = []
    for generic in (1, 0):
        v = fg.default_variant()
        v.az_generic = generic
        b = fg.Batch([(params, planets)], fg.FARGO_FP32_BULK, variant=v)
        d = b.disk(0)
        d.set_fields(**f)
        d.substep(fg.SUB_TRANSPORT, dt)
        got.append(d.field("dens")[:-1])
        b.close()
    assert not np.array_equal(got[0], f["dens"][:-1])
    off = float((got[0] != got[1]).mean())
    print("cells that differ: %.5f" % off)
    assert off < 0.01
