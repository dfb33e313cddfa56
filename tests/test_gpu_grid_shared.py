"""rg_deposit_ngp with one grid given for several properties: the properties add up in it, then it is
clamped and divided once for each of them, in their order.

Deposits on whole numbers below 2^24 are exact in float whatever the order of the atomics, and the
divisors are powers of two, so the results are exact."""

import numpy as np
import pytest

import grid_oracle as go
import rg_b200 as rg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 48, 128])
@pytest.mark.parametrize("owner,divisors", [
    ([0, 0], [2.0, 4.0]),
    ([0, 0], None),
    ([0, 1, 0], [1.0, 2.0, 8.0]),          # the first use divides by nothing, a negative property between
    ([0, 1, 1, 0, 2], [0.5, 4.0, 1.0, 2.0, 2.0]),
])
def test_shared_grids_finish_in_order(n, owner, divisors):
    import torch
    rng = np.random.default_rng(n + len(owner))
    box, ng, n_prop = 1.3 * n, 200 * n, len(owner)
    pos = (rng.random((ng, 3)) * box).astype(np.float32)
    vals = rng.integers(-3, 9, (n_prop, ng)).astype(np.float32)
    vals[0] = np.abs(vals[0])
    grids = [torch.full((n * n * (n + 2),), 7.0, device="cuda") for _ in range(max(owner) + 1)]
    dpos, dval = (torch.from_numpy(a.ravel().copy()).cuda() for a in (pos, vals))
    torch.cuda.synchronize()
    ctx = rg.Context(n)
    ctx.deposit_ngp(box, ng, dpos.data_ptr(), dval.data_ptr(), [grids[o].data_ptr() for o in owner], divisors)
    ctx.close()
    cell = tuple(go.pos_to_ngp(pos[:, a], box, n) for a in range(3))
    for o, g in enumerate(grids):
        mine = [p for p in range(n_prop) if owner[p] == o]
        want = np.zeros((n, n, n + 2))
        for p in mine:
            np.add.at(want, cell, vals[p].astype(np.float64))
        for p in mine:
            want = np.maximum(want, 0.0) / (divisors[p] if divisors else 1.0)
        assert np.array_equal(g.cpu().numpy().reshape(n, n, n + 2), want), o
