"""The FP32 march of the source step, the viscosities and the energy equation (k_gas, for disks
that run beside a million cells) against the kernels with one thread per cell that a
small disk alone takes.  Both call the same arithmetic, written with rounding intrinsics, so the
fields have to be bitwise equal: over whole DTs and over the substeps' parts, with
columns of less, exactly and more than a block's (120), chunks with a remainder, rings fewer
than a chunk, every boundary, self-gravity, a rotating frame, and no planet.
"""
import numpy as np
import pytest

import cudaprotoplanetarydisks_gb300 as fg
from tests.helpers import small

pytestmark = pytest.mark.gpu
FIELDS = ("dens", "vrad", "vtheta", "energy", "pressure", "temperature", "divergence", "qplus")

CASES = [("c1", 8, 9, {}), ("c1", 33, 119, {}), ("c3", 16, 120, {}), ("c3", 17, 121, {}), ("c3", 35, 260, dict(cooling=0)),
         ("c2", 16, 96, {}), ("c2", 24, 144, dict(adiabatic=1)), ("c3", 20, 64, dict(nb=0)), ("c1", 19, 50, dict(open_inner=1)),
         ("c3", 21, 70, dict(open_inner=1)), ("c3", 24, 100, dict(non_reflecting=1)), ("c3", 30, 90, dict(evanescent=1)),
         ("c3", 40, 129, dict(corotating=1)), ("c1", 18, 66, dict(imposeddiskdrift=1e-3))]


def pair(cfg, nrad, nsec, extra):
    params, planets = small(cfg, nrad=nrad, nsec=nsec, **{k: v for k, v in extra.items() if k != "nb"})
    if "nb" in extra:
        planets = []
    big = small("c1", nrad=1000, nsec=1000)
    alone = fg.Disk(params, planets, fg.FARGO_FP32_BULK)
    return alone, fg.Batch([(params, planets), big], fg.FARGO_FP32_BULK)


def kernels(d):
    import ctypes
    ms, n = (ctypes.c_double * 96)(), ctypes.c_int(0)
    assert d.lib.fargo_time_substep_kernels(d.h, 1, ms, 96, ctypes.byref(n)) == 0
    return [d.lib.fargo_substep_kernel_name(d.h, k).decode() for k in range(n.value)]


@pytest.mark.parametrize("cfg,nrad,nsec,extra", CASES)
def test_gas_march_is_bitwise_the_cell_kernels(cfg, nrad, nsec, extra):
    alone, batch = pair(cfg, nrad, nsec, extra)
    d = batch.disk(0)
    for _ in range(2):
        assert alone.step_DT() == d.step_DT()
        for k in FIELDS:
            assert np.array_equal(alone.field(k), d.field(k)), k
    for which in (fg.SUB_POTENTIAL, fg.SUB_SOURCE) + ((fg.SUB_ENERGY,) if cfg == "c3" else ()) + (fg.SUB_TRANSPORT,):
        for x in (alone, d):
            x.substep(which, 1e-3)
        for k in FIELDS:
            assert np.array_equal(alone.field(k), d.field(k)), (which, k)
    for x in (alone, d):
        x.substep_full(1e-3)
    for k in FIELDS:
        assert np.array_equal(alone.field(k), d.field(k)), k
    assert "k_source" in kernels(alone) and "k_gas" in kernels(d)
    batch.close()
