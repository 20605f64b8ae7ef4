"""Read-out of the statistics with the device's memory used up: it needs none, and gives the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fill_device(torch):
    """Allocations that leave little of the device free."""
    held, size = [], 1 << 36
    while size >= 1 << 21:
        try:
            held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            size //= 2
    return held


def test_readout_without_device_memory(built):
    import torch
    torch.cuda.empty_cache()
    # a context of its own: its pool holds no freed block that the read-out could take. The values of
    # the plane statistics are 107 MB, those of the profiles 5 MB.
    ctx = built.Context(0)
    L, lx, ly = 400, 20, 3000
    mask = np.full((ly, lx), 125, np.uint8)
    mask[1:-1, 1:-1] = 0
    dom = built.make_domain(lx, ly, L, mask=mask, radius=8.0, buffer_depth=3)
    s = built.Solve(ctx, dom, built.Params.make(tblend=0.5, pin=0.01, nu=0.02, delta=2, blend=1.0), built.F32)
    s.init_poiseuille(0.1, noise=0.01, seed=3)
    for _ in range(2):
        s.step(1)
        s.stats_sample()
        s.profile_sample()
    s.sync()
    held = fill_device(torch)
    try:
        assert torch.cuda.mem_get_info()[0] < 1 << 26
        full, prof = s.stats_get(), s.profile_get()
    finally:
        held.clear()
        torch.cuda.empty_cache()
    free, prof_free = s.stats_get(), s.profile_get()
    assert full[1:] == free[1:] == (2, 2) and prof[1] == prof_free[1] == 2
    assert full[0].any() and np.array_equal(full[0], free[0])
    assert prof[0].any() and np.array_equal(prof[0], prof_free[0])
    s.close()
    ctx.close()
