"""ComputeTs' X-ray sums by x_e nodes for every way a number of nodes is taken (odd counts, whose last
Lyman-alpha field has a unit of its own; one to four chunks of k_ts_nodes, of two, three and four nodes),
against the oracle.  Each case says how many nodes it is to run by, from rg_debug_ts_nodes, so that a
change of the rule cannot empty it.

The rule weighs a node against the shells' passes: of the cases of test_gpu_ts_nodes.py the two that span
one interval of the table run by nodes and the others by shells.

Tolerances as in the other ComputeTs comparisons (1e-5): the sums differ from the by-shell ones only in
where they are rounded."""

import numpy as np
import pytest

import rg_b200 as rg
import test_gpu_ts as tt
import test_gpu_ts_agn as ta
import test_gpu_ts_nodes as tn
import ts_oracle as to
import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ts_tables():
    return to.TsTables()


def x_e_range(tab, nodes):
    """x_e from the table's first node to its interval nodes - 2."""
    X = np.asarray(tab.X, np.float64)
    lo = 1.05 * X[0]
    hi = max(1.5 * lo, min(1.02 * X[nodes - 2], 0.9985))
    return float(np.float32(lo)), float(np.float32(hi))


def ran_by(p, zz, idx, x_e):
    return rg.ts_nodes(p, zz, idx, idx + 1, float(x_e.min()), float(x_e.max()))[1:3]


@pytest.mark.parametrize("nodes,chunks,ftype,shells", [
    (2, 1, 0, 40), (3, 1, 2, 40), (4, 1, 0, 40), (5, 2, 0, 40), (6, 2, 2, 40), (7, 2, 0, 40), (8, 2, 0, 40),
    (9, 3, 2, 40), (3, 1, 1, 40), (5, 2, 1, 62), (7, 2, 1, 62), (10, 3, 0, 62), (13, 4, 0, 62), (14, 4, 2, 62),
])
def test_number_of_nodes(ts_tables, nodes, chunks, ftype, shells):
    n = 16
    lo, hi = x_e_range(ts_tables, nodes)
    zz, idx, src, ti = tn.case(n, 1100 + nodes + shells, lo, hi)
    p = rg.make_params(n, 1.5 * n, Flag_IncludeSpinTemp=1, TsHeatingFilterType=ftype, TsNumFilterSteps=shells)
    assert ran_by(p, zz, idx, wl.from_padded(ti.x_e_box_prev)) == (nodes, chunks)
    out, res = tt.run_gpu_ts(p, zz, idx, src, ti)
    want, wg = tt.run_oracle_ts(p, ts_tables, zz, idx, src, ti)
    tt.check_parity(out, res, want, wg, n)


@pytest.mark.parametrize("nodes,chunks,ftype,flag", [(3, 1, 0, 1), (5, 2, 2, 2), (9, 3, 0, 1), (3, 1, 1, 3), (0, 0, 1, 1)])
def test_agn_bands_next_to_nodes(ts_tables, nodes, chunks, ftype, flag):
    n = 16
    lo, hi = x_e_range(ts_tables, nodes or 12)
    zz, idx, src, ti = tn.case(n, 1200 + nodes + flag, lo, hi)
    agn = ta.agn_inputs(src, ti, 1250 + flag)
    p = rg.make_params(n, 1.5 * n, Flag_IncludeSpinTemp=1, TsHeatingFilterType=ftype, Flag_IncludeAGNXray=flag)
    assert ran_by(p, zz, idx, wl.from_padded(ti.x_e_box_prev)) == (nodes, chunks)
    out, res = ta.run_gpu(p, zz, idx, src, ti, agn)
    want, wg = ta.run_oracle(p, ts_tables, zz, idx, src, ti, agn)
    tt.check_parity(out, res, want, wg, n)
    for k in ("volume_ave_Xheat_AGN_soft", "volume_ave_Xheat_AGN_hard"):
        assert abs(getattr(out, k) - want[k]) <= 1e-5 * abs(want[k]) + 1e-300, k
