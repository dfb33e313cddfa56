"""ComputeTs with its X-ray sums formed in k-space by x_e nodes, and by shells where the box's x_e
spans too many nodes, against the oracle.

The sums differ from the by-shell ones only in where they are rounded (FP32, each term to 2^-24 of
the largest), so the tolerances are those of the other ComputeTs comparisons (1e-5)."""

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


def case(n, seed, lo, hi):
    zz, idx = wl.snapshot_redshifts(12.0)
    src = wl.make_sources(n, 1.5 * n, seed)
    ti = wl.make_ts_inputs(src, zz, idx, idx + 1, seed + 1)
    rng = np.random.default_rng(seed + 2)
    xe = np.exp(rng.uniform(np.log(lo), np.log(hi), (n, n, n))).astype(np.float32)
    xe.flat[0], xe.flat[1] = lo, hi
    ti.x_e_box_prev = wl.to_padded(xe)
    return zz, idx, src, ti


@pytest.mark.parametrize("n,lo,hi,shells,ftype", [
    (16, 4.677e-4, 4.677e-4, 40, 1),    # the whole box on one node: two nodes
    (16, 1e-6, 1.5e-4, 7, 0),           # below the table (clamped): 6 fields of 7 shells, window table
    (32, 0.991, 1.0, 40, 1),            # the last interval and above the table (clamped)
    (32, 1.1e-4, 2e-3, 16, 1),          # five nodes: 15 fields of 16 shells
    (32, 1.1e-4, 2e-3, 15, 1),          # the same nodes, 15 shells: by shells
    (32, 1e-5, 0.9999, 40, 2),          # all nodes, by shells, window table
    (64, 1e-5, 0.9999, 43, 1),          # all nodes: 42 fields of 43 shells (an odd count)
    (8, 1e-4, 1e-2, 40, 1),             # the smallest grid
])
def test_xray_sums_match_oracle(ts_tables, n, lo, hi, shells, ftype):
    zz, idx, src, ti = case(n, 900 + n + shells, lo, hi)
    p = rg.make_params(n, 1.5 * n, Flag_IncludeSpinTemp=1, TsHeatingFilterType=ftype, TsNumFilterSteps=shells)
    out, res = tt.run_gpu_ts(p, zz, idx, src, ti)
    want, wg = tt.run_oracle_ts(p, ts_tables, zz, idx, src, ti)
    tt.check_parity(out, res, want, wg, n)


@pytest.mark.parametrize("lo,hi,flag", [(1e-4, 3e-3, 1), (1e-5, 0.9999, 1), (1e-5, 0.9999, 2), (1e-4, 1e-3, 3)])
def test_agn_units_next_to_nodes_and_shells(ts_tables, lo, hi, flag):
    n = 32
    zz, idx, src, ti = case(n, 950 + flag, lo, hi)
    agn = ta.agn_inputs(src, ti, 955 + flag)
    p = rg.make_params(n, 1.5 * n, Flag_IncludeSpinTemp=1, Flag_IncludeAGNXray=flag)
    out, res = ta.run_gpu(p, zz, idx, src, ti, agn)
    want, wg = ta.run_oracle(p, ts_tables, zz, idx, src, ti, agn)
    tt.check_parity(out, res, want, wg, n)
    for k in ("volume_ave_Xheat_AGN_soft", "volume_ave_Xheat_AGN_hard"):
        assert abs(getattr(out, k) - want[k]) <= 1e-5 * abs(want[k]) + 1e-300, k
