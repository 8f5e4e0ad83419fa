"""The FP32 march of the source step, the viscosities and the energy equation (k_gas) with every kind of chunk that a
rule on the disk's size can give it, from 4 rings to 64, against the kernels with one thread per cell: bitwise
equal fields over whole DTs.  Among the disks a rotating frame beside each boundary (the frame's change inside the march,
the boundary beside the planets' update, the edge rings' energy afterwards), and the fused form of an
ensemble of a million cells.
"""
import ctypes

import numpy as np
import pytest

import cudaprotoplanetarydisks_gb300 as fg
from cudaprotoplanetarydisks_gb300 import _capi
from tests.helpers import small

pytestmark = pytest.mark.gpu
FIELDS = ("dens", "vrad", "vtheta", "energy", "pressure", "temperature", "divergence", "qplus")


def marched(params, planets, rings):
    """The disk with k_gas in chunks of `rings` rings, whatever its size."""
    lib = _capi.load()
    f, p = lib.fargo_ctx_create_among, ctypes.c_void_p
    f.argtypes = [ctypes.POINTER(fg.FargoParams), ctypes.POINTER(fg.FargoPlanet), ctypes.c_int, ctypes.c_int, p, p,
                  ctypes.c_longlong, ctypes.c_int, ctypes.POINTER(p)]
    h = p()
    assert f(ctypes.byref(params), (fg.FargoPlanet * max(1, len(planets)))(*planets), len(planets), fg.FARGO_FP32_BULK, None, None, 0,
             rings, ctypes.byref(h)) == 0
    return fg.Disk(params, planets, fg.FARGO_FP32_BULK, _handle=h)


def kernels(d):
    ms, n = (ctypes.c_double * 96)(), ctypes.c_int(0)
    assert d.lib.fargo_time_substep_kernels(d.h, 1, ms, 96, ctypes.byref(n)) == 0
    return [d.lib.fargo_substep_kernel_name(d.h, k).decode() for k in range(n.value)]


CASES = [("c1", 35, 119, {}), ("c3", 70, 121, {}), ("c3", 66, 240, dict(corotating=1)), ("wide", 67, 130, {}),
         ("c3", 39, 122, dict(corotating=1, evanescent=1)), ("c1", 41, 90, dict(corotating=1, open_inner=1)),
         ("c3", 43, 90, dict(corotating=1, open_inner=1)), ("c2", 48, 96, dict(adiabatic=1))]


@pytest.mark.parametrize("rings", [4, 5, 17, 64])
@pytest.mark.parametrize("cfg,nrad,nsec,extra", CASES)
def test_chunks(cfg, nrad, nsec, extra, rings):
    params, planets = small(cfg, nrad=nrad, nsec=nsec, **extra)
    alone, d = fg.Disk(params, planets, fg.FARGO_FP32_BULK), marched(params, planets, rings)
    for _ in range(2):
        assert alone.step_DT() == d.step_DT()
        for k in FIELDS:
            assert np.array_equal(alone.field(k), d.field(k)), k
        assert [(p.x, p.y, p.vx, p.vy) for p in alone.planets()] == [(p.x, p.y, p.vx, p.vy) for p in d.planets()]
    assert "k_source" in kernels(alone) and "k_gas" in kernels(d)
    d.lib.fargo_ctx_destroy(d.h)
    d.h = None
    alone.close()


def test_fused_ensemble_of_a_million_cells():
    members = [small("c1", nrad=1000, nsec=1000), small("c3", nrad=40, nsec=120), small("c1", nrad=33, nsec=244),
               small("c3", nrad=50, nsec=300, corotating=1), small("c1", nrad=20, nsec=64, corotating=1)]
    batch = fg.Batch(members, fg.FARGO_FP32_BULK).fuse()
    for _ in range(2):
        batch.run_async(1)
        batch.sync()
    for (params, planets), d in zip(members, batch.disks):
        alone = fg.Disk(params, planets, fg.FARGO_FP32_BULK)
        for _ in range(2):
            alone.step_DT()
        # (the other four depend on whether the DT ended with a substep of dt = 0, which only a disk alone has)
        for k in FIELDS[:4]:
            assert np.array_equal(alone.field(k), d.field(k)), (params.nrad, k)
        alone.close()
    assert any(k == "kb_gas" for k, _ in batch.fused_kernel_times(1))
    batch.close()
