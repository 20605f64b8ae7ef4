"""The step's split over the SMs (tile height, streamwise chunks) at the edges of its range: short
pipes, odd plane counts (a chunk's last pair of planes is half used), cross-sections that end
inside a tile, with the seam's pressure jump, a force and the gauge. Against the FP64 oracle at
the suite's FP32 bound (1e-5 relative L2; 1e-12 for FP64), and bit for bit between tile heights:
a cell's arithmetic does not depend on the split."""
import numpy as np
import pytest

import oracle_lib as O
from test_gpu_parity import circle_mask, errors, run_gpu

pytestmark = pytest.mark.gpu

# (L, lx, ly): shortest pipe, one tile and one pair per chunk, odd everything, several tiles
SIZES = [(5, 9, 9), (6, 33, 20), (33, 24, 41), (64, 65, 40), (151, 61, 61)]


def case(L, lx, ly):
    m2 = circle_mask(lx, ly, min(lx, ly) / 2 - 1, (lx - 1) / 2, (ly - 1) / 2)
    rng = np.random.default_rng(1000 * L + lx)
    f = np.zeros((4, L, ly, lx))
    f[0] = 1e-3 * rng.uniform(-1, 1, f[0].shape)
    f[1:] = 0.02 * rng.uniform(-1, 1, f[1:].shape)
    f[3] -= 0.05
    f *= m2 == 0
    f = f.astype(np.float32).astype(np.float64)
    prm = dict(tblend=0.5, pin=0.002, nu=0.03, d1=2, blend=1.0, force=(1e-6, 2e-6, -5e-6))
    return m2, f, prm


@pytest.mark.parametrize("L,lx,ly", SIZES)
def test_tile_heights_match_oracle_and_each_other(built, ctx, monkeypatch, L, lx, ly):
    m2, f, prm = case(L, lx, ly)
    dom = built.make_domain(lx, ly, L, mask=m2, radius=min(lx, ly) / 2 - 1, buffer_depth=4)
    steps = 7
    ref, _ = O.run_core(m2, L, f, prm, steps, monitor_every=3, radius=min(lx, ly) / 2 - 1)
    for dtype in (built.F32, built.F16):
        outs = []
        for ty in ("0", "8", "16", "32"):          # 0: the library's choice
            monkeypatch.setenv("FSLBM_TILE_Y", ty)
            outs.append(run_gpu(built, ctx, dom, prm, dtype, f, steps, monitor_every=3)[0])
        for o in outs[1:]:
            assert np.array_equal(outs[0], o)
        if dtype == built.F32:
            _, eu, eps = errors(outs[0], ref, m2)
            assert eu <= 1e-5 and eps <= 1e-5, (eu, eps)
    outs = []
    for ty in ("0", "8", "16"):
        monkeypatch.setenv("FSLBM_TILE_Y", ty)
        outs.append(run_gpu(built, ctx, dom, prm, built.F64, f, steps, monitor_every=3)[0])
    for o in outs[1:]:
        assert np.array_equal(outs[0], o)
    _, eu, eps = errors(outs[0], ref, m2)
    assert eu <= 1e-12 and eps <= 1e-12, (eu, eps)


@pytest.mark.parametrize("order,rough", [(6, False), (0, True), (6, True)])
@pytest.mark.parametrize("L,lx,ly", [(7, 33, 20), (33, 24, 41), (40, 65, 40)])
def test_three_taps_and_masks_per_plane(built, ctx, monkeypatch, L, lx, ly, order, rough):
    """The pair kernel's 3-tap corrector and its masks per plane, every tile height it has, with
    wall bumps that start and end inside a pair of planes and on the seam."""
    m2, f, prm = case(L, lx, ly)
    mask = m2
    if rough:
        mask = np.repeat(m2[None], L, axis=0)
        inner = np.argwhere(m2 == 0)
        for z in (0, 3, L - 1):                   # a few fluid cells of these planes become wall
            for y, x in inner[z % 5::7]:
                mask[z, y, x] = 125
        f = f * (mask == 0)
    prm = dict(prm, fd_order=order, blend=0.4 if order == 6 else 1.0)
    dom = built.make_domain(lx, ly, L, mask=mask, radius=min(lx, ly) / 2 - 1, buffer_depth=4)
    steps = 7
    ref, _ = O.run_core(mask, L, f, prm, steps, monitor_every=0)
    outs = []
    for ty in ("0", "8", "16") + (("32",) if order == 0 else ()):
        monkeypatch.setenv("FSLBM_TILE_Y", ty)
        outs.append(run_gpu(built, ctx, dom, prm, built.F32, f, steps, monitor_every=0)[0])
    for o in outs[1:]:
        assert np.array_equal(outs[0], o)
    fluid = (mask == 0) if rough else np.broadcast_to(mask == 0, f[0].shape)
    d, want = (outs[0] - ref)[:, fluid], ref[:, fluid]
    scale = np.abs(want[0]) + 1.5 * (want[1:] ** 2).sum(0)
    assert np.linalg.norm(d[1:]) <= 1e-5 * np.linalg.norm(want[1:])
    assert np.linalg.norm(d[0]) <= 1e-5 * np.linalg.norm(scale)
    assert not outs[0][:, ~fluid].any()
