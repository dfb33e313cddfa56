"""find_HII_bubbles on a device with little room: the radii go in smaller batches, with the same results;
where not even one radius fits the call returns RG_ENOMEM and the context stays usable.

The memory is taken by the test before the call (plain allocations that fail are errors of the API, not
faults).  At 128^3 with two grids 16 radii take 273 MB, their windows 19 MB, the spectra 17 MB."""

import numpy as np
import pytest

import rg_b200 as rg
import test_gpu_hii_paths as tp
import workloads as wl

pytestmark = pytest.mark.gpu

N, MB = 128, 1 << 20


class Taken:
    """All but `left` to `left` + 10 MB of the device."""

    def __init__(self, left):
        self.left, self.parts = left, []

    def __enter__(self):
        import torch
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        while True:
            # from 10 MB on a tensor is an allocation of its own, of its size in steps of 2 MB
            size = min(1 << 36, (torch.cuda.mem_get_info()[0] - self.left) // (2 * MB) * (2 * MB))
            if size < 10 * MB:
                return self
            self.parts.append(torch.empty(size, dtype=torch.uint8, device="cuda"))

    def __exit__(self, *exc):
        import torch
        self.parts.clear()
        torch.cuda.empty_cache()


def call(ctx, dg, p):
    import ctypes as C
    zz, snap = wl.snapshot_redshifts(8.0)
    s = rg.snapshot(zz, snap)
    out = rg.rg_hii_scalars()
    ctx.call("rg_find_HII_bubbles", C.byref(p), C.byref(s), C.byref(dg.g), C.byref(out))
    return out


def fresh(seed):
    return tp.case(N, seed, False, False, False, 0)


@pytest.mark.parametrize("left", [320 * MB, 294 * MB, 200 * MB, 64 * MB])
def test_smaller_batches_give_the_same(left):
    want, p = fresh(5)
    ref = rg.Context(N)
    o = call(ref, want, p)           # loads the kernels too
    ref.close()
    a, _ = fresh(5)
    b, _ = fresh(5)
    ctx = rg.Context(N)
    with Taken(left):
        got = [call(ctx, a, p), call(ctx, b, p)]     # the second with the size that fitted
    ctx.close()
    for dg, g in zip((a, b), got):
        assert g.as_dict() == o.as_dict()
        for k in tp.OUT:
            assert np.array_equal(dg.get(k), want.get(k)), k


def test_no_room_is_enomem_and_the_context_stays_usable():
    want, p = fresh(6)
    ref = rg.Context(N)
    o = call(ref, want, p)
    ref.close()
    a, _ = fresh(6)
    ctx = rg.Context(N)
    with Taken(12 * MB):
        with pytest.raises(rg.RGError) as e:
            call(ctx, a, p)
        assert e.value.status == rg.RG_ENOMEM
    ctx.profile(True)
    assert call(ctx, a, p).as_dict() == o.as_dict()
    # with the default batch again, not one that was tried where nothing fitted
    passes = {s["name"]: s["launches"] for s in ctx.kernel_stats()}["inv_xy_c2c_window"]
    ctx.close()
    assert passes == -(-o.n_radii // 16)
    for k in tp.OUT:
        assert np.array_equal(a.get(k), want.get(k)), k


def test_a_set_batch_that_does_not_fit_is_enomem():
    want, p = fresh(7)
    ref = rg.Context(N)
    o = call(ref, want, p)
    ref.close()
    a, _ = fresh(7)
    ctx = rg.Context(N)
    ctx.call("rg_set_radius_batch", 16)
    with Taken(200 * MB):
        with pytest.raises(rg.RGError) as e:
            call(ctx, a, p)
        assert e.value.status == rg.RG_ENOMEM
        ctx.call("rg_set_radius_batch", 4)
        assert call(ctx, a, p).as_dict() == o.as_dict()
    ctx.close()


def test_a_failed_allocation_does_not_reach_later_calls():
    import ctypes as C

    import torch
    n = 32
    p = rg.make_params(n, float(n), Flag_IncludeSpinTemp=1)
    ctx = rg.Context(n)
    g = rg.rg_grids()
    with pytest.raises(rg.RGError) as e:
        ctx.call("rg_alloc_grids", C.byref(p), 2_000_000, C.byref(g))    # 278 GB a history grid
    assert e.value.status == rg.RG_ENOMEM
    x = torch.ones(n * n * (n + 2), device="cuda")
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    ctx.call("rg_debug_filter_roundtrip", C.byref(p), x.data_ptr(), y.data_ptr(), 3.0, -1)
    ctx.close()
    assert torch.allclose(y.view(n, n, n + 2)[:, :, :n], torch.ones(n, n, n, device="cuda"), atol=1e-5)
