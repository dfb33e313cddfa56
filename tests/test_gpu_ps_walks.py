"""The power spectrum's bins with walks of 2 (48^3), 4 (96^3) and 32 (192^3) modes along x, and of a
box whose columns leave most of a block idle (8^3), against the oracle; tolerances of test_gpu_ps.py."""

import numpy as np
import pytest

import ps_oracle as po
import rg_b200 as rg
from test_gpu_ps import close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 48, 96, 192])
def test_bins_match_oracle(n):
    import torch
    rng = np.random.default_rng(n + 17)
    dT = (15.0 + 4.0 * rng.standard_normal((n, n, n))).astype(np.float32)
    p = rg.make_params(n, 0.9 * n, Hubble_h=0.7)
    ctx = rg.Context(n)
    d = torch.from_numpy(dT.ravel()).cuda()
    k, ps, err = ctx.power_spectrum(p, d.data_ptr())
    ctx.close()
    wk, wps, werr, _ = po.power_spectrum(dT, 0.9 * n, 0.7)
    assert len(k) == len(wk)
    assert close(k, wk, 1e-6)
    assert close(ps, wps, 1e-5)
    assert close(err, werr, 1e-5)
