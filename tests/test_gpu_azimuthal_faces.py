"""The FP64 azimuthal transport's interfaces (k_transport_azimuthal_warp).  Two warps form the flux of the
interface between them, and what leaves one has to be bit for bit what enters the other, also where only
one of them holds a cell whose value the float pairs do not take (below 2^-40) or whose density is so low that
rho / (rho + 1e-20) is not 1.  So no cell's result may depend on which warp it falls to: a ring
turned by some sectors gives the result turned by them.  (Velocities are multiples of 2^-20, whose mean is exact in any
order; without radial velocities the radial transport leaves everything as it is.)
"""
import numpy as np
import pytest

import cudaprotoplanetarydisks_gb300 as fg
from tests.helpers import small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsec", [128, 480, 603])
@pytest.mark.parametrize("kind", ["ordinary", "small energies", "low densities", "both"])
def test_turned_rings(nsec, kind):
    params, planets = small("c3", nrad=16, nsec=nsec)
    rng = np.random.default_rng(nsec)
    shape = (params.nrad + 1, nsec)
    f = dict(dens=params.sigma0 * rng.uniform(0.5, 1.5, shape), vrad=np.zeros(shape),
             vtheta=np.round((1.0 + 0.02 * rng.normal(size=shape)) * 2 ** 20) / 2 ** 20,
             energy=params.sigma0 * 1e-3 * rng.uniform(0.5, 1.5, shape))
    if kind in ("small energies", "both"):
        f["energy"][rng.random(shape) < 0.01] = 1e-20
    if kind in ("low densities", "both"):
        f["dens"][rng.random(shape) < 0.01] = 3e-5
    for v in f.values():
        v[-1] = 0.0
    dt = 0.25 * 2 * np.pi / nsec * params.rmin / 0.1
    d = fg.Disk(params, planets, fg.FARGO_FP64)

    def transport(turn):
        d.set_fields(**{k: np.roll(v, turn, axis=1) for k, v in f.items()})
        d.substep(fg.SUB_TRANSPORT, dt)
        return {k: np.roll(d.field(k), -turn, axis=1) for k in f}

    want = transport(0)
    assert not np.array_equal(want["dens"], f["dens"])
    for turn in (1, 4, 37, 60, 119):
        got = transport(turn)
        for k in f:
            assert np.array_equal(got[k], want[k]), (turn, k)
    d.close()
