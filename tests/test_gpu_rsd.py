"""The line-of-sight re-binning by itself (sizes whose lines do not fill a block, displacements of many
cells and around the box, sub-cells that cross or spread), and the deposit into grids that are not
16-byte aligned.

The oracle's re-binning (FP64 sums) gets the device's own delta_T of flag 2, which is what flag 3
re-bins, so the FP32 gradient before it, ill-conditioned where dv/dz is near -H, does not enter.  A cell
sums up to a few hundred float shares in any order: 2^-24 of the shares' absolute values each time a
sum is rounded, well below 1e-6 of the norm of those absolute values."""

import ctypes as C

import numpy as np
import pytest

import grid_oracle as go
import rg_b200 as rg
import vel_oracle as vo
import workloads as wl
from helpers import DeviceGrids, oracle_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,amp,rough", [(24, 20.0, 0.0), (48, 600.0, 0.0), (96, 200.0, 0.0), (64, 0.0, 0.0),
                                         (32, 5000.0, 0.0), (32, 0.0, 40.0), (48, 100.0, 15.0), (128, 40.0, 2.0)])
def test_rebinning_matches_oracle(n, amp, rough):
    import torch
    rng = np.random.default_rng(n)
    box = 1.25 * n
    xH = rng.random((n, n, n)).astype(np.float32)
    xH[rng.random((n, n, n)) < 0.3] = 0.0
    deltax = wl.to_padded((0.3 * rng.standard_normal((n, n, n))).astype(np.float32))
    TS = (20.0 + 80.0 * rng.random((n, n, n))).astype(np.float32)
    # a shift per line, a small wave along it, and rough: differences of cell widths from cell to cell, so
    # that sub-cells cross in about a third of the cells
    vel = np.repeat(amp * rng.standard_normal((n, n, 1)), n, axis=2)
    vel += 2.0 * np.sin(2 * np.pi * np.arange(n) / n)
    vel += rough * rng.standard_normal((n, n, n))
    vel = wl.to_padded(vel.astype(np.float32))
    zz, snap = wl.snapshot_redshifts(8.0)
    s = rg.snapshot(zz, snap)
    dv = torch.from_numpy(vel.ravel()).cuda()
    ctx = rg.Context(n)
    got = {}
    for flag in (2, 3):
        p = rg.make_params(n, box, Flag_IncludeSpinTemp=1, Flag_IncludePecVelsFor21cm=flag)
        dg = DeviceGrids(n, spin=True)
        for k, v in (("deltax", deltax), ("xH", xH), ("TS_box", TS)):
            dg.put(k, v)
        dg.g.vel = dv.data_ptr()
        tb = C.c_double()
        ctx.call("rg_delta_T", C.byref(p), C.byref(s), C.byref(dg.g), C.byref(tb))
        got[flag] = dg.get("delta_T")
    ctx.close()
    z = float(zz[snap])
    vc = vo.convert_velocity(vel[:, :, :n], 0, z)
    H_z = np.float32(vo.hubble(oracle_params(p), z))
    want = vo.rsd(got[2], xH, vc, H_z, box / p.Hubble_h)
    scale = np.linalg.norm(vo.rsd(np.abs(got[2]), xH, vc, H_z, box / p.Hubble_h))
    assert np.linalg.norm(got[3].astype(np.float64) - want) <= 1e-6 * scale
    assert tb.value == pytest.approx(float(got[3].astype(np.float64).mean()), rel=1e-9, abs=1e-12 * scale)


@pytest.mark.parametrize("shift", [0, 1, 3])
def test_deposit_into_unaligned_grids(shift):
    import torch
    n, box, ng = 24, 30.0, 5000
    rng = np.random.default_rng(shift)
    pos = (rng.random((ng, 3)) * box).astype(np.float32)
    vals = rng.lognormal(0, 1, (3, ng)).astype(np.float32)
    vals[1] -= 1.0
    npad = n * n * 2 * (n // 2 + 1)
    buf = torch.full((3, npad + 4), 7.0, dtype=torch.float32, device="cuda")
    dpos, dval = torch.from_numpy(pos.ravel()).cuda(), torch.from_numpy(vals.ravel()).cuda()
    div = [1.0, 1.0, 3.0]
    ctx = rg.Context(n)
    ctx.deposit_ngp(box, ng, dpos.data_ptr(), dval.data_ptr(), [buf[p].data_ptr() + 4 * shift for p in range(3)], div)
    ctx.close()
    got = buf.cpu().numpy()
    want = go.deposit_ngp(n, box, pos, vals, div)
    absg = go.deposit_ngp(n, box, pos, np.abs(vals), div)
    for p in range(3):
        assert np.all(np.abs(got[p, shift:shift + npad].reshape(want[p].shape) - want[p]) <= 1e-5 * absg[p] + 1e-30)
        assert np.all(got[p, :shift] == 7.0) and np.all(got[p, shift + npad:] == 7.0)   # nothing around it
