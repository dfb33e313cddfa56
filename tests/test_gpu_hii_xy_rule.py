"""The fused x/y pass on either side of each line of its rule (plan and blocks an SM by size and grids an
item) against the plain mode, and a batch that crosses the line against its snapshots: the same bits, as
the plans run the same butterflies in the same order."""

import numpy as np
import pytest

import rg_b200 as rg
import test_gpu_hii_paths as tp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,spin,bh", [
    (24, False, False), (48, False, False), (48, True, True), (96, True, False), (96, True, True),
    (192, False, False), (192, True, False), (64, False, False), (64, True, False), (128, False, False),
    (128, True, False), (256, False, False), (256, False, True)])
def test_each_side_of_the_rule_equals_plain_mode(n, spin, bh):
    a, p = tp.case(n, 170 + n, spin, bh, False, 0)
    b, _ = tp.case(n, 170 + n, spin, bh, False, 0)
    oa = tp.run(n, a, p, rg.RG_MODE_FUSED, 5)
    ob = tp.run(n, b, p, rg.RG_MODE_PLAIN)
    assert 0.0 < oa.volume_weighted_global_xH < 1.0
    for k in tp.OUT:
        assert np.array_equal(a.get(k), b.get(k)), k
    assert oa.as_dict() == ob.as_dict()


@pytest.mark.parametrize("n,units", [(48, 3), (96, 3), (192, 3), (64, 2), (256, 2)])
def test_batch_across_the_line_equals_single_snapshots(n, units):
    tp.test_batch_equals_single_snapshots(n, units, False)
