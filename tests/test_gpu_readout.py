"""Read-out of the statistics (combined on the device): before any sample, after a reset of the
fluctuation sums, and on a width that is not a multiple of the device pitch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lx,L", [(21, 7), (24, 30)])
def test_readout(built, ctx, lx, L):
    c = (lx - 1) / 2
    dom = built.make_domain(lx, lx, L, radius=lx / 2 - 1, cx=c, cy=c, buffer_depth=3)
    s = built.Solve(ctx, dom, built.Params.make(tblend=0.5, pin=0.01, nu=0.02, delta=2, blend=1.0), built.F64)
    s.init_poiseuille(0.1, noise=0.01, seed=3)
    st, c1, c2 = s.stats_get()
    pr, n = s.profile_get()
    assert not st.any() and not pr.any() and (c1, c2, n) == (0, 0, 0)
    means, prof = [], np.zeros((10, lx, lx))
    for k in range(3):
        s.step(1)
        if k == 2:                                   # restart the fluctuation sums only
            s.set_params(built.Params.make(tblend=0.5, pin=0.01, nu=0.02, delta=1, blend=1.0))
        s.stats_sample()
        s.profile_sample()
        q, u, v, w = f = s.get_fields()
        means.append(f[:, :, :, lx // 2])            # (4, L, ly)
        prof += np.array([a.sum(0) for a in (q, u, v, w, u * u, v * v, w * w, u * v, u * w, v * w)])
    st, c1, c2 = s.stats_get()
    assert (c1, c2) == (3, 1)
    core = st.reshape(11, L + 6, lx)[:, 3:-3]
    mean = np.mean(means, axis=0)
    assert np.abs(core[:4] - mean).max() <= 1e-14    # three additions and a division of values below 1
    dev = mean - means[-1]
    assert np.abs(core[4:8] - np.abs(dev)).max() <= 1e-14
    assert np.abs(core[8] - dev[1] * dev[2]).max() <= 1e-15
    pr, n = s.profile_get()
    assert n == 3 and np.abs(pr - prof).max() <= 1e-12 * max(1.0, np.abs(prof).max())
    s.close()
