"""The two plans of ComputeTs' z pass, with the X-ray sums by nodes and by shells, with and without AGN
bands, against the oracle.  The box is an 8^3 field repeated 16 (32) times, whose result is the 8^3 one
repeated (test_gpu_tiled.py); tolerances as there (1e-5)."""

from types import SimpleNamespace

import numpy as np
import pytest

import rg_b200 as rg
import test_gpu_ts as tt
import test_gpu_ts_agn as ta
import ts_oracle as to
import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ts_tables():
    return to.TsTables()


# the one-exchange plan by nodes without AGN bands, and by shells at 256^3; else 8 values a thread
@pytest.mark.parametrize("reps,nodes,flag", [(16, 3, 0), (16, 0, 0), (16, 3, 1), (16, 0, 1), (32, 0, 0)])
def test_z_pass_plans(ts_tables, reps, nodes, flag):
    n = 8
    zz, idx = wl.snapshot_redshifts(15.0)
    src = wl.make_sources(n, 8.0, 1300)
    ti = wl.make_ts_inputs(src, zz, idx, 16, 1301)
    X = np.asarray(ts_tables.X, np.float64)
    lo, hi = (float(np.float32(v)) for v in (1.05 * X[0], 1.02 * X[(nodes or 12) - 2]))
    xe = np.exp(np.random.default_rng(1302).uniform(np.log(lo), np.log(hi), (n, n, n))).astype(np.float32)
    xe.flat[0], xe.flat[1] = lo, hi
    ti.x_e_box_prev = wl.to_padded(xe)
    agn = ta.agn_inputs(src, ti, 1303)
    kw = dict(Flag_IncludeSpinTemp=1, Flag_IncludeAGNXray=flag)
    p8, p = rg.make_params(n, 8.0, **kw), rg.make_params(n * reps, 8.0 * reps, **kw)
    assert rg.ts_nodes(p, zz, idx, 16, float(xe.min()), float(xe.max()))[1] == nodes
    real = lambda a: np.tile(np.asarray(a).reshape(n, n, n), (reps, reps, reps))
    pad = lambda a: wl.to_padded(real(wl.from_padded(np.asarray(a).reshape(n, n, -1))))
    big = SimpleNamespace(n=n * reps, **{k: pad(getattr(src, k)) for k in ("deltax", "stars", "sfr", "xray")})
    bti = SimpleNamespace(x_e_box_prev=pad(ti.x_e_box_prev), Tk_box=real(ti.Tk_box),
                          sfr_histories=[pad(a) for a in ti.sfr_histories],
                          xray_histories=[pad(a) for a in ti.xray_histories], stored_fcoll=ti.stored_fcoll)
    if flag:
        bagn = {k: [pad(a) for a in v] if isinstance(v, list) else pad(v) for k, v in agn.items()}
        out, res = ta.run_gpu(p, zz, idx, big, bti, bagn)
        want, wg = ta.run_oracle(p8, ts_tables, zz, idx, src, ti, agn)
    else:
        out, res = tt.run_gpu_ts(p, zz, idx, big, bti)
        want, wg = tt.run_oracle_ts(p8, ts_tables, zz, idx, src, ti)
    tiled = {k: real(wg[k]) for k in ("x_e_box_prev", "x_e_box", "Tk_box", "TS_box")}
    tt.check_parity(out, res, want, tiled, n * reps)
