"""How ComputeTs chooses to form its X-ray sums (by x_e nodes or shell by shell), and that what k_ts_nodes
reads of a shell's coefficients lies in the shell's array, for every number of nodes (host only)."""

import numpy as np
import pytest

import rg_b200 as rg
import workloads as wl

XE_LO = 1.1e-4   # on the table's first node
# upper ends of x_e that reach each further node of the table
XE_HI = (1.2e-4, 3e-4, 5e-4, 2e-3, 3e-3, 5e-3, 1e-2, 3e-2, 5e-2, 0.1, 0.3, 0.6, 0.9, 0.95, 0.99, 0.9999)


def choose(n, ftype, shells, lo, hi):
    zz, idx = wl.snapshot_redshifts(12.0)
    p = rg.make_params(n, 1.5 * n, Flag_IncludeSpinTemp=1, TsHeatingFilterType=ftype, TsNumFilterSteps=shells)
    return rg.ts_nodes(p, zz, idx, idx + 1, lo, hi)


@pytest.mark.parametrize("ftype", [0, 1, 2])
@pytest.mark.parametrize("shells", [15, 40, 62, 110, 400])
def test_coefficients_read_lie_in_the_shells_array(ftype, shells):
    counts = set()
    for hi in XE_HI:
        m0, nm, chunks, reads, held = choose(16, ftype, shells, XE_LO, hi)
        counts.add(nm)
        if nm == 0:
            assert chunks == reads == 0
            continue
        assert 0 <= m0 and 2 <= nm and m0 + nm <= 14
        assert chunks >= 1 and 3 * nm <= reads <= held
    if shells == 400:
        assert counts >= {2, 3, 4, 5, 7, 8, 10, 11, 12, 13, 14}
    if shells == 15 and ftype == 1:
        assert counts == {0}


def test_nan_keeps_the_shells():
    assert choose(16, 0, 400, XE_LO, float(np.float32("nan")))[1] == 0
    assert choose(16, 0, 400, XE_LO, XE_LO)[1] == 2
