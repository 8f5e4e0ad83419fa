"""The fields that only the last substep of a DT writes (pressure, temperature, divergence and, with the
energy equation, Q+) after a DT that fails in a substep which looked like an ordinary one when it
began.  They belong to that substep, not to an earlier DT.
"""
import numpy as np
import pytest

import cudaprotoplanetarydisks_gb300 as fg
from tests.helpers import small

pytestmark = pytest.mark.gpu
PREC = [fg.FARGO_FP64, fg.FARGO_FP32_BULK]


def moved(d):
    """The disk's fields at twice the density and energy and with another radial velocity."""
    f = {k: d.field(k) for k in ("dens", "vrad", "vtheta", "energy")}
    f["dens"] = 2 * f["dens"]
    f["energy"] = 2 * f["energy"]
    f["vrad"][2:-2] += 1e-3
    return f


def check_fresh(d, before, dens, energy, soundspeed):
    # of the given density and energy but for a substep's change: an earlier DT's would be off by half
    dens, p = dens[:-1], d.field("pressure")[:-1]
    own = 0.4 * energy[:-1] if energy is not None else dens * soundspeed[:-1] ** 2
    with np.errstate(invalid="ignore", divide="ignore"):
        assert np.nanmedian(np.abs(p / own - 1)) < 0.02
    assert (d.field("divergence")[2:-2] != before["divergence"][2:-2]).mean() > 0.9
    if energy is not None:
        assert (d.field("qplus")[2:-2] != before["qplus"][2:-2]).mean() > 0.9


# a density that is not finite, which the disk's force on the star shows before the substep, and two empty
# cells, whose pressure gradient (0/0) is only found after it
@pytest.mark.parametrize("prec", PREC)
@pytest.mark.parametrize("cfg,extra,pad,bad", [("c1", dict(open_inner=1), 1, np.nan), ("c1", {}, 0, np.nan), ("c3", {}, 0, np.inf),
                                               ("c3", dict(open_inner=1), 1, np.inf), ("c1", {}, 0, 0.0), ("c1", dict(open_inner=1), 1, 0.0)])
def test_diagnostics_after_a_failed_dt(cfg, extra, pad, bad, prec):
    params, planets = small(cfg, nrad=40, nsec=120, **extra)
    v = fg.default_variant()
    v.pad = pad
    b = fg.Batch([(params, planets)], prec, variant=v)
    d = b.disk(0)
    assert d.step_DT() > 2
    before = {k: d.field(k) for k in ("pressure", "temperature", "divergence", "qplus")}
    f = moved(d)
    f["dens"][5, 7:9] = bad
    d.set_fields(**f)
    with pytest.raises(fg.FargoError, match="non-finite density"):
        d.step_DT()
    assert not np.isfinite(d.field("temperature")[5, 7])
    if cfg == "c1" and bad != 0.0:
        p = d.field("pressure")
        assert np.array_equal(np.isfinite(p), np.isfinite(f["dens"]))
    check_fresh(d, before, f["dens"], f["energy"] if cfg == "c3" else None, d.field("soundspeed"))
    b.close()
