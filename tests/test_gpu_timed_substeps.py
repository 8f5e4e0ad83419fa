"""The fields that only the last substep of a DT writes (pressure, temperature, divergence and, with the
energy equation, Q+) after substeps that are run to be timed: of the last one, not of an earlier DT.
"""
import ctypes

import numpy as np
import pytest

import cudaprotoplanetarydisks_gb300 as fg
from tests.helpers import small
from tests.test_gpu_failed_dt import PREC, moved

pytestmark = pytest.mark.gpu
FIELDS = ("pressure", "temperature", "divergence", "qplus")


def check(d, before, adiabatic):
    dens, p = d.field("dens")[:-1], d.field("pressure")[:-1]
    own = 0.4 * d.field("energy")[:-1] if adiabatic else dens * d.field("soundspeed")[:-1] ** 2
    # an earlier DT's would be off by half
    assert np.median(np.abs(p / own - 1)) < 0.02
    assert np.median(np.abs(d.field("temperature")[:-1] * dens / own - 1)) < 0.02
    for k in FIELDS[2:] if adiabatic else FIELDS[2:3]:
        assert (d.field(k)[2:-2] != before[k][2:-2]).mean() > 0.9, k


@pytest.mark.parametrize("prec", PREC)
@pytest.mark.parametrize("reps", [1, 3])
@pytest.mark.parametrize("cfg", ["c1", "c3"])
def test_one_disk(cfg, reps, prec):
    params, planets = small(cfg, nrad=40, nsec=120)
    d = fg.Disk(params, planets, prec)
    d.step_DT()
    before = {k: d.field(k) for k in FIELDS}
    d.set_fields(**moved(d))
    ms, n = (ctypes.c_double * 96)(), ctypes.c_int(0)
    assert d.lib.fargo_time_substep_kernels(d.h, reps, ms, 96, ctypes.byref(n)) == 0
    check(d, before, cfg == "c3")
    d.close()


@pytest.mark.parametrize("prec", PREC)
def test_a_fused_batch(prec):
    b = fg.Batch([small("c1", nrad=40, nsec=120), small("c3", nrad=40, nsec=120)], prec).fuse()
    b.run_async(1)
    b.sync()
    before = [{k: d.field(k) for k in FIELDS} for d in b.disks]
    for d in b.disks:
        d.set_fields(**moved(d))
    b.fused_kernel_times(2)
    for d, was, adiabatic in zip(b.disks, before, (False, True)):
        check(d, was, adiabatic)
    b.close()
