"""The frequency tables that the device integrates for ComputeTs against the host engine's.

Both run the same adaptive rule in FP64; the integrands interpolate the electron tables in float,
where the device fuses a multiply and an add that the host rounds twice: two float roundings, so
every table entry agrees to 2 x 2^-23 = 2.4e-7 relative (5e-7 with the cross sections' own FP64
rounding and a node that rounds to the neighbouring float energy)."""

import ctypes as C

import numpy as np
import pytest

import rg_b200 as rg
import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("z,shells,agn,x_e,fcoll", [
    (8.0, 1, 0, 2e-4, 1e-3),        # one shell
    (15.0, 40, 1, 2e-4, 1e-3),      # both AGN bands
    (6.5, 33, 2, 0.6, 2e-2),        # mostly ionised gas, the hard band
    (12.0, 15, 3, 0.99995, 1e-6),   # above the x_e where nu_tau_one is not sought, the soft band
    (35.0, 8, 0, 1e-3, 0.0),        # early: no collapsed gas
])
def test_device_frequency_tables_match_host_engine(z, shells, agn, x_e, fcoll):
    zz, snap = wl.snapshot_redshifts(z)
    p = rg.make_params(32, 64.0, Flag_IncludeSpinTemp=1, TsNumFilterSteps=shells, Flag_IncludeAGNXray=agn)
    prev = np.zeros(len(zz))
    prev[snap - 1] = 0.7 * fcoll
    _, freq, _ = rg.ts_tables(p, zz, snap, snap + 1, x_e, fcoll, prev)
    bands, _ = rg.ts_agn_tables(p, zz, snap, snap + 1, x_e, fcoll, prev)
    want = np.concatenate([freq[None], bands])
    got = np.full_like(want, np.nan)
    s = rg.snapshot(zz, snap, prev)
    ctx = rg.Context(32)
    ctx.call("rg_debug_ts_device_tables", C.byref(p), C.byref(s), snap + 1, x_e, fcoll, shells, got.ctypes.data)
    ctx.close()
    assert np.any(want[0] > 0)
    assert np.all(np.abs(got - want) <= 5e-7 * np.abs(want))
