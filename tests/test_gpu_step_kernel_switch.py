"""FSLBM_STEP_KERNEL=1 runs the general one-column kernel where the pair and FP64 column kernels are the
library's choice: against the oracle at the suite's bounds (1e-5 relative L2 for FP32, 1e-12 for FP64)."""
import numpy as np
import pytest

import oracle_lib as O
from test_gpu_parity import errors, run_gpu
from test_gpu_splits import case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,order", [("F32", 0), ("F32", 6), ("F64", 0)])
@pytest.mark.parametrize("L,lx,ly", [(7, 33, 20), (33, 24, 41)])
def test_general_kernel(built, ctx, monkeypatch, dt, order, L, lx, ly):
    monkeypatch.setenv("FSLBM_STEP_KERNEL", "1")
    m2, f, prm = case(L, lx, ly)
    prm = dict(prm, fd_order=order, blend=0.4 if order else 1.0)
    radius = min(lx, ly) / 2 - 1
    dom = built.make_domain(lx, ly, L, mask=m2, radius=radius, buffer_depth=4)
    ref, _ = O.run_core(m2, L, f, prm, 7, monitor_every=3, radius=radius)
    got, _ = run_gpu(built, ctx, dom, prm, getattr(built, dt), f, 7, monitor_every=3)
    _, eu, eps = errors(got, ref, m2)
    tol = 1e-5 if dt == "F32" else 1e-12
    assert eu <= tol and eps <= tol, (eu, eps)
    assert not got[:, :, m2 != 0].any()
