"""Batches that cannot give every SM an item at 8 planes per chunk march chunks down to a pair of
planes; odd lengths, lengths of one chunk and cross-sections that end just inside a second tile, with
both tile heights and all warp shapes. A member's fields and monitor records equal the solve stepped
alone bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (L, n) of the members: one tile and one pair of planes per chunk, odd everything, second tiles with
# two rows or columns, 16 equal pipes (4 planes per chunk)
BATCHES = [[(5, 9)], [(8, 24)], [(33, 33), (7, 20)], [(64, 48)], [(61, 36), (40, 68)], [(32, 24)] * 16]


def make(built, ctx, L, n, dtype, seed):
    s = built.Solve(ctx, built.make_domain(n, n, L, radius=n / 2 - 1, buffer_depth=4),
                    built.Params.make(tblend=0.5, pin=0.002, nu=0.03, d1=2, blend=1.0, monitor_every=3,
                                      force=(1e-6, 2e-6, -5e-6)), dtype)
    s.init_poiseuille(0.1, noise=1e-2, seed=seed)
    return s


@pytest.mark.parametrize("dt", ["F32", "F16"])
@pytest.mark.parametrize("sizes", BATCHES, ids=lambda b: f"{len(b)}x{b[0][0]}x{b[0][1]}")
def test_equal_to_members_alone(built, ctx, monkeypatch, dt, sizes):
    dtype, steps = getattr(built, dt), 7
    alone = []
    for k, (L, n) in enumerate(sizes):
        s = make(built, ctx, L, n, dtype, k)
        s.step(steps)
        s.sync()
        alone.append((s.get_fields(np.float32), s.monitor_log()))
        s.close()
    for tile_y in (None, "16", "32"):              # None: the library's choice
        if tile_y:
            monkeypatch.setenv("FSLBM_BATCH_TILE_Y", tile_y)
        members = [make(built, ctx, L, n, dtype, k) for k, (L, n) in enumerate(sizes)]
        b = built.Batch(ctx, members)
        for i in range(len(members)):
            b.set_tiling(i, 256, i % 3 if len(members) > 1 else 1)
        b.step(steps)
        b.sync()
        for s, (want, log) in zip(members, alone):
            assert np.array_equal(s.get_fields(np.float32), want)
            got = s.monitor_log()
            assert [r["step"] for r in got] == [3, 6]
            for g, w in zip(got, log):
                assert all(g[key] == w[key] for key in ("q1", "p1", "p2", "sample"))
        b.close()
        for s in members:
            s.close()
