"""Parameters that need a longer tile list than memory is left for: set_params fails, the solve is not
stepped with the list that it no longer has, and setting the same parameters again makes it whole."""
import numpy as np
import pytest

from test_gpu_readout_memory import fill_device

pytestmark = pytest.mark.gpu


def test_set_params_without_device_memory(built):
    import torch
    torch.cuda.empty_cache()
    # a wide, short box: 65536 tiles of 32 x 8 for the general kernel, 512 KB, more than the largest piece
    # (the monitor log, 320 KB) that the small solves below leave
    lx = ly = 4096
    L = 20
    mask = np.full((ly, lx), 125, np.uint8)
    mask[1:-1, 1:-1] = 0
    dom = built.make_domain(lx, ly, L, mask=mask, radius=8.0, buffer_depth=3)

    def params(order):
        return built.Params.make(tblend=0.5, pin=0.0, nu=0.02, delta=2, blend=1.0, fd_order=order)

    ctx = built.Context(0)
    s = built.Solve(ctx, dom, params(0), built.F32)
    s.init_poiseuille(0.1, noise=0.01, seed=3)
    s.step(1)
    s.sync()
    held, small = fill_device(torch), []
    try:
        small_dom = built.make_domain(24, 24, 16, radius=11.0, buffer_depth=3)
        with pytest.raises(built.FslbmError):          # the pool's last blocks, in small pieces
            for _ in range(4000):
                small.append(built.Solve(ctx, small_dom, params(0), built.F32))
        try:
            s.set_params(params(8))                    # may fit where a larger piece is left
        except built.FslbmError:
            with pytest.raises(built.FslbmError, match="set_params failed"):
                s.step(1)
        s.sync()
    finally:
        held.clear()
        for q in small:
            q.close()
        torch.cuda.empty_cache()
    s.set_params(params(8))
    s.step(1)
    s.sync()
    got = s.get_plane(1, 3), s.check()
    s.close()

    s = built.Solve(ctx, dom, params(0), built.F32)
    s.init_poiseuille(0.1, noise=0.01, seed=3)
    s.step(1)
    s.set_params(params(8))
    s.step(1)
    s.sync()
    assert got[0].any()
    assert np.array_equal(got[0], s.get_plane(1, 3)) and got[1] == s.check()
    s.close()
    ctx.close()
