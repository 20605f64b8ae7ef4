"""Host starts through the server's reused buffers: requests of growing, shrinking and equal sizes,
one burst after the other, each with its own start; results equal the same solve run alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(40, 24), (33, 41), (64, 32), (40, 24), (16, 24)]      # (L, n)


def test_bursts_of_host_starts(built, ctx):
    fb = built

    def setup(L, n, seed):
        c = (n - 1) / 2
        dom = fb.make_domain(n, n, L, radius=n / 2 - 1, cx=c, cy=c)
        prm = fb.Params.make(tblend=0.5, pin=0.0, nu=0.02, blend=1.0, force=(0.0, 0.0, -1e-5))
        f = fb.init_poiseuille(dom, 0.1, noise=0.05, seed=seed).astype(np.float32)
        return dom, prm, f

    with fb.Server(0) as srv:
        for burst in range(3):
            reqs = [setup(L, n, 10 * burst + i) for i, (L, n) in enumerate(SIZES)]
            ids = [srv.submit(d, p, fb.F32, 7 + burst, init=f) for d, p, f in reqs]
            for _, _, f in reqs:
                f[:] = np.nan                      # the server holds its own copy
            srv.drain(60.0)
            for i, (rid, (L, n)) in enumerate(zip(ids, SIZES)):
                assert srv.poll(rid)["status"] == fb.REQ_DONE
                dom, prm, f = setup(L, n, 10 * burst + i)
                s = fb.Solve(ctx, dom, prm, fb.F32)
                s.set_fields(f)
                s.step(7 + burst)
                want = s.get_fields(np.float32)
                s.close()
                assert np.array_equal(srv.release(rid), want)
