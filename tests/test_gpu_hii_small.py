"""find_HII_bubbles below 64^3: the z pass compiled for its number of grids against the one that reads it at
run time.

Pop III sources that are zero everywhere take the same call through the run-time form (one more grid,
whose terms add zeros), so every output has the same bits; J_21 with black-hole feedback is a sum of two
products, of which either may be fused with the addition: two roundings, 2 x 2^-24 relative."""

import numpy as np
import pytest

import rg_b200 as rg
import test_gpu_hii_paths as tp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 16, 24, 32, 48])
@pytest.mark.parametrize("spin,bh", [(False, False), (True, False), (False, True), (True, True)])
def test_grid_count_at_compile_time_equals_run_time(n, spin, bh):
    got, p = tp.case(n, 40 + n, spin, bh, False, 0)
    want, q = tp.case(n, 40 + n, spin, bh, False, 0)
    zero = [got.torch.zeros_like(want.t["stars"]) for _ in range(2)]
    want.g.starsIII, want.g.weighted_sfrIII = (z.data_ptr() for z in zero)
    q.UseMiniHalos = 1
    q.ReionNionPhotPerBaryIII = q.ReionNionPhotPerBary
    q.ReionEfficiencyIII = q.ReionEfficiency
    a = tp.run(n, got, p, rg.RG_MODE_FUSED, 5)
    b = tp.run(n, want, q, rg.RG_MODE_FUSED, 5)
    assert 0.0 < a.volume_weighted_global_xH < 1.0
    for k in tp.OUT:
        if k == "J_21_at_ionization" and bh:
            x, y = got.get(k).astype(np.float64), want.get(k).astype(np.float64)
            assert np.all(np.abs(x - y) <= 2.0 ** -23 * np.abs(y))
        else:
            assert np.array_equal(got.get(k), want.get(k)), k
    assert a.as_dict() == b.as_dict()
