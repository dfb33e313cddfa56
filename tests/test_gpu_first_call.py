"""A context's first call gives what its later calls give: the tables it uploads are on the device before
the kernels that read them start."""

import ctypes as C

import numpy as np
import pytest

import rg_b200 as rg
import workloads as wl

pytestmark = pytest.mark.gpu


def frequency_tables(ctx, x_e, shells=8):
    zz, snap = wl.snapshot_redshifts(12.0)
    p = rg.make_params(16, 24.0, Flag_IncludeSpinTemp=1, TsNumFilterSteps=shells)
    s = rg.snapshot(zz, snap, np.zeros(len(zz)))
    out = np.full((3, 3, 14, shells), np.nan)
    ctx.call("rg_debug_ts_device_tables", C.byref(p), C.byref(s), snap + 1, x_e, 1e-6, shells, out.ctypes.data)
    return out


# above x_e = 0.9999 nu_tau_one is not sought, so the kernels that read the electron tables come at once
@pytest.mark.parametrize("x_e", [0.99995, 2e-4])
def test_first_frequency_tables_equal_later_ones(x_e):
    for _ in range(8):
        ctx = rg.Context(16)
        first = frequency_tables(ctx, x_e)
        again = frequency_tables(ctx, x_e)
        ctx.close()
        assert np.any(first[0] > 0)
        assert np.array_equal(first, again)


def roundtrip(ctx, n, d_in, d_out):
    p = rg.make_params(n, float(n))
    ctx.call("rg_debug_filter_roundtrip", C.byref(p), d_in.data_ptr(), d_out.data_ptr(), 3.0, 0)
    return d_out.clone()


@pytest.mark.parametrize("n", [8, 96, 128])
def test_first_transform_equals_later_ones(n):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(n)
    d_in = torch.randn(n * n * (n + 2), generator=gen, device="cuda")
    d_out = torch.zeros_like(d_in)
    torch.cuda.synchronize()
    for _ in range(8):
        ctx = rg.Context(n)
        first = roundtrip(ctx, n, d_in, d_out)
        again = roundtrip(ctx, n, d_in, d_out)
        ctx.close()
        assert torch.equal(first, again)
