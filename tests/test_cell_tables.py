"""Masks per plane: the solve holds one table of wall sums, of the kernel that steps it, in a buffer
that serves either kernel. The memory is that of the larger table (16 bytes per cell for FP32), and a
change of parameters that moves the solve between the kernels gives what a new solve gives."""
import ctypes

import numpy as np
import pytest

import oracle_lib as O
from test_gpu_masks3d import rough_case
from test_gpu_parity import errors, run_gpu


@pytest.mark.parametrize("dt,state,table", [("F32", 4, 16), ("F64", 8, 32)])
def test_footprint(built, dt, state, table):
    L, n = 64, 96
    dom = built.make_domain(n, n, L, mask=np.full((L, n, n), 125, np.uint8), radius=40.0)
    b = ctypes.c_int64()
    built._check(built.lib().fslbm_solve_footprint(ctypes.byref(dom), getattr(built, dt), ctypes.byref(b)))
    cells = n * n * L
    small = b.value - cells * (2 * 4 * state + 1 + table)       # tile list, monitor log
    assert 0 < small < 1 << 20, small


def params(d1, order):
    """d1 = 1 at nu = 0.12, as in the corrector-order tests: at 0.03 that stride is unstable (the oracle's
    fields grow to 1e123 within 20 steps)."""
    return dict(tblend=0.8, pin=0.002, nu=0.12 if d1 == 1 else 0.03, d1=d1, fd_order=order,
                blend=0.4 if order else 1.0, force=(0.0, 0.0, -1e-5))


@pytest.mark.gpu
@pytest.mark.parametrize("dt,d1,order", [("F32", 1, 0), ("F32", 2, 8), ("F32", 3, 0), ("F64", 1, 0)])
def test_one_column_kernel(built, ctx, dt, d1, order):
    """The general kernel with masks per plane where the pair kernel does not run, against the oracle
    at the suite's bounds (1e-5 relative L2 for FP32, 1e-12 for FP64)."""
    m3, n, L, R, f, _ = rough_case()
    prm = params(d1, order)
    dom = built.make_domain(n, n, L, mask=m3, radius=R, buffer_depth=4)
    ref, _ = O.run_core(m3, L, f, prm, 20, monitor_every=0)
    got, _ = run_gpu(built, ctx, dom, prm, getattr(built, dt), f, 20)
    _, eu, eps = errors(got, ref, np.where(np.all(m3 == 0, axis=0), 0, 125))
    tol = 1e-5 if dt == "F32" else 1e-12
    assert eu <= tol and eps <= tol, (eu, eps)
    assert not got[:, m3 != 0].any()


@pytest.mark.gpu
@pytest.mark.parametrize("order", [0, 6])
def test_pair_kernel_against_one_column(built, ctx, monkeypatch, order):
    """Both kernels compute the same step; each is within 1e-5 of the oracle, so within 2e-5 of the other."""
    m3, n, L, R, f, _ = rough_case()
    prm = params(2, order)
    dom = built.make_domain(n, n, L, mask=m3, radius=R, buffer_depth=4)
    pair, _ = run_gpu(built, ctx, dom, prm, built.F32, f, 20)
    monkeypatch.setenv("FSLBM_STEP_KERNEL", "1")
    col, _ = run_gpu(built, ctx, dom, prm, built.F32, f, 20)
    _, eu, eps = errors(pair, col, np.where(np.all(m3 == 0, axis=0), 0, 125))
    assert eu <= 2e-5 and eps <= 2e-5, (eu, eps)


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["F32", "F64"])
def test_change_of_kernel(built, ctx, dt):
    m3, n, L, R, f, _ = rough_case()
    dom = built.make_domain(n, n, L, mask=m3, radius=R, buffer_depth=4)
    dtype = getattr(built, dt)
    s = built.Solve(ctx, dom, built.Params.make(**params(2, 0)), dtype)
    held, b = s.info()["bytes_device"], ctypes.c_int64()
    built._check(built.lib().fslbm_solve_footprint(ctypes.byref(dom), dtype, ctypes.byref(b)))
    assert held <= b.value
    for d1, order in ((2, 0), (1, 0), (2, 6 if dt == "F32" else 0), (1, 0), (2, 0)):
        prm = params(d1, order)
        s.set_params(built.Params.make(**prm))
        s.set_fields(f)
        s.step(5)
        s.sync()
        assert s.info()["bytes_device"] <= b.value + f.nbytes      # set_fields' staging of the host type
        want, _ = run_gpu(built, ctx, dom, prm, dtype, f, 5)
        assert np.array_equal(s.get_fields(), want), (d1, order)
    s.close()
