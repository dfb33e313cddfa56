"""The forms of find_HII_bubbles' passes give the same bits.

The fused x/y pass, the two-pass form of the plain mode, the z pass on registers and the row-buffer
one run the same butterflies in the same order on the same float windows, and the barrier test is the
same FP64 expression, so every grid of the fused mode equals the plain mode's (one radius per batch,
no fused pass), and a snapshot of a batch equals its own call."""

import ctypes as C

import numpy as np
import pytest

import rec_oracle as rco
import rg_b200 as rg
import workloads as wl
from helpers import DeviceGrids

pytestmark = pytest.mark.gpu

OUT = ("xH", "r_bubble", "z_at_ionization", "J_21_at_ionization", "temp_kinetic_all_gas")
REC = ("Gamma12", "N_rec", "residual_xH", "clumping_factor", "t_resp")


def case(n, seed, spin, bh, rec, ftype):
    rng = np.random.default_rng(seed)
    src = wl.make_sources(n, float(n), seed)
    dg = DeviceGrids(n, spin=spin, bh=bh, rec=rec)
    for k, v in (("deltax", src.deltax), ("stars", src.stars), ("weighted_sfr", src.sfr)):
        dg.put(k, v)
    if spin:
        dg.put("x_e_box", wl.to_padded((0.2 * rng.random((n, n, n))).astype(np.float32)))
        dg.put("Tk_box", (10.0 + 990.0 * rng.random((n, n, n))).astype(np.float32))
    if bh:
        dg.put("effective_bhm", (src.stars * 0.05 * rng.random(src.stars.shape)).astype(np.float32))
        dg.put("effective_bhar", (src.sfr * 0.3 * rng.random(src.sfr.shape)).astype(np.float32))
    if rec:
        dg.put("N_rec", wl.to_padded((0.3 * rng.random((n, n, n))).astype(np.float32)))
    p = rg.make_params(n, float(n), Flag_EvolvingReionRBubbleMax=0, ReionRBubbleMax=20.0, ReionRBubbleMaxRecomb=20.0,
                       ReionEfficiency=12000.0, ReionFilterType=ftype, Flag_IncludeSpinTemp=int(spin),
                       Flag_BHFeedback=int(bh), Flag_IncludeRecombinations=int(rec), ReionUVBFlag=2 if rec else 1)
    # some cells were ionised before this snapshot
    z0 = np.where(rng.random((n, n, n)) < 0.1, 9.5, -1.0).astype(np.float32)
    dg.put("z_at_ionization", z0)
    return dg, p


def run(n, dg, p, mode, batch=0):
    zz, snap = wl.snapshot_redshifts(8.0)
    s = rg.snapshot(zz, snap)
    ctx = rg.Context(n)
    ctx.call("rg_set_mode", mode)
    ctx.call("rg_set_radius_batch", batch)
    if p.Flag_IncludeRecombinations:
        t = rco.synthetic_tables()
        ctx.set_recombination_tables(t.knots, *(t.y[k].reshape(t.nz, t.nt, t.ng) for k in range(3)))
    out = rg.rg_hii_scalars()
    ctx.call("rg_find_HII_bubbles", C.byref(p), C.byref(s), C.byref(dg.g), C.byref(out))
    ctx.close()
    return out


@pytest.mark.parametrize("n,spin,bh,rec,ftype", [
    (24, True, False, False, 0), (64, True, True, False, 0), (64, False, True, True, 1), (96, True, True, True, 0),
    (96, False, False, False, 2), (128, True, False, True, 0), (128, True, True, True, 2), (192, True, True, False, 0),
    (192, False, False, True, 0), (256, True, True, True, 0), (384, False, True, False, 1)])
def test_fused_mode_equals_plain_mode(n, spin, bh, rec, ftype):
    a, p = case(n, 70 + n, spin, bh, rec, ftype)
    b, _ = case(n, 70 + n, spin, bh, rec, ftype)
    oa = run(n, a, p, rg.RG_MODE_FUSED, 5)     # batches that end off the schedule's length
    ob = run(n, b, p, rg.RG_MODE_PLAIN)
    assert 0.0 < oa.volume_weighted_global_xH < 1.0
    for k in OUT + (REC if rec else ()):
        assert np.array_equal(a.get(k), b.get(k)), k
    assert oa.as_dict() == ob.as_dict()
    assert not np.any(np.signbit(a.get("xH")))


@pytest.mark.parametrize("n,units,bh", [(96, 2, True), (96, 7, True), (64, 10, False), (24, 3, False), (192, 2, False)])
def test_batch_equals_single_snapshots(n, units, bh):
    ones = [case(n, 300 + u, False, bh, False, 0) for u in range(units)]
    many = [case(n, 300 + u, False, bh, False, 0) for u in range(units)]
    so = [run(n, dg, p, rg.RG_MODE_FUSED) for dg, p in ones]
    zz, snap = wl.snapshot_redshifts(8.0)
    s = [rg.snapshot(zz, snap) for _ in many]
    ctx = rg.Context(n)
    mo = ctx.find_hii_batch([p for _, p in many], s, [dg.g for dg, _ in many])
    ctx.close()
    for (a, _), (b, _), oa, ob in zip(ones, many, so, mo):
        for k in OUT:
            assert np.array_equal(a.get(k), b.get(k)), k
        assert oa.as_dict() == ob.as_dict()
