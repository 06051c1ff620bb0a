"""CGLS on plans whose projections all run on the tensor cores (48 slices and more):
the tolerance stop, warm starts with their denominator, the best iterate's return and the
statistical weights, against the oracle in double.

A result may be as far from FP64 as the reference's float solve, or 1e-5: 5 steps amplify
rounding by 1e2 to 1e3 (the reference's own residuals are 7e-8 off after four steps and
1e-6 to 7e-6 after five).  Of a warm start only the result is held to that: its residual
b - A x0 is a difference of nearly equal numbers, a hundredth of either.
"""
import numpy as np
import pytest

from conftest import rel_l2, uniform_angles
from devutil import empty_vol, sino_to_dev, vol_from_dev, vol_to_dev

pytestmark = pytest.mark.gpu

CASES = [(3, 65, 48, 64, 1), (2, 65, 56, 72, 2)]


def problem(gb, oc, w, nx, ny, na, seed, scale=1.0):
    ang, rng = uniform_angles(na), np.random.default_rng(seed)
    plan = gb.Plan(w, 0.5 * (nx - 1), ny, ang)
    with oc.op_threads():
        b = oc.project(w, 0.5 * (nx - 1), rng.random((plan.nrays, ny), dtype=np.float32) * np.float32(scale), ang)
    return plan, ang, (b + 0.01 * rng.standard_normal(b.shape)).astype(np.float32)


def close(x, hist, x64, h64, x_ref, h_ref, trace=True):
    print("from FP64: here %.1e, the reference %.1e; residuals off by %s" % (
        rel_l2(x, x64), rel_l2(x_ref, x64), np.abs(np.asarray(hist) / np.asarray(h64) - 1)))
    assert rel_l2(x, x64) < max(1e-5, 1.1 * rel_l2(x_ref, x64))
    if not trace:
        return
    h, h64, h_ref = np.asarray(hist), np.asarray(h64), np.asarray(h_ref)
    assert h.shape == h64.shape
    assert np.abs(h / h64 - 1).max() < max(1e-5, 1.1 * np.abs(h_ref / h64 - 1).max())


@pytest.mark.parametrize("w,nx,ny,na,seed", CASES)
def test_tolerance_stop(gb, oc, w, nx, ny, na, seed):
    plan, ang, b = problem(gb, oc, w, nx, ny, na, seed)
    with oc.op_threads():
        _, t = oc.cgls64(w, b, ang, maxit=5, tol=0.0)
        tol = float(np.sqrt(t.rel_history()[3] * t.rel_history()[4]))
        x64, t64 = oc.cgls64(w, b, ang, maxit=20, tol=tol)
        x_ref, t_ref = oc.cgls(w, b, ang, maxit=20, tol=tol)
    assert t64.iterations == t_ref.iterations == 5
    xd = empty_vol(plan)
    hist, info = plan.cgls(sino_to_dev(plan, b), xd, 20, tol)
    assert info.iterations == 5 and info.iterbest == t64.iterbest
    close(vol_from_dev(plan, xd), hist, x64, t64.rel_history(), x_ref, t_ref.rel_history())
    assert plan.check() == 0


@pytest.mark.parametrize("w,nx,ny,na,seed", CASES)
def test_warm_start_and_its_denominator(gb, oc, w, nx, ny, na, seed):
    plan, ang, b = problem(gb, oc, w, nx, ny, na, seed)
    with oc.op_threads():
        x0, t0 = oc.cgls64(w, b, ang, maxit=2, tol=0.0)
        x0 = x0.astype(np.float32)
        x64, t64 = oc.cgls64(w, b, ang, maxit=4, tol=0.0, x0=x0, rnorm_ref=t0.rnorm0)
        x_ref, t_ref = oc.cgls(w, b, ang, maxit=4, tol=0.0, x0=x0, rnorm_ref=t0.rnorm0)
    xd = vol_to_dev(plan, x0)
    hist, info = plan.cgls(sino_to_dev(plan, b), xd, 4, 0.0, warm=True, rnorm_ref=t0.rnorm0)
    assert info.iterations == 4
    close(vol_from_dev(plan, xd), hist, x64, t64.rel_history(), x_ref, t_ref.rel_history(), trace=False)


def test_best_iterate_is_given_back(gb, oc):
    """The third step's residual is above the second's, whose iterate comes back."""
    w, nx, ny, na, seed = CASES[0]
    plan, ang, b = problem(gb, oc, w, nx, ny, na, seed)
    with oc.op_threads():
        x64, t64 = oc.cgls64(w, b, ang, maxit=4, tol=0.0)
        x3, t3 = oc.cgls64(w, b, ang, maxit=3, tol=0.0)
        x_ref, t_ref = oc.cgls(w, b, ang, maxit=3, tol=0.0)
    assert t3.rel_history()[2] > t3.rel_history()[1]
    xd = empty_vol(plan)
    hist, info = plan.cgls(sino_to_dev(plan, b), xd, 3, 0.0)
    assert info.iterbest == t3.iterbest
    close(vol_from_dev(plan, xd), hist, x3, t3.rel_history(), x_ref, t_ref.rel_history())


@pytest.mark.parametrize("warm", [False, True])
@pytest.mark.parametrize("w,nx,ny,na,seed", CASES)
def test_statistical_weights(gb, oc, w, nx, ny, na, seed, warm):
    plan, ang, b = problem(gb, oc, w, nx, ny, na, seed, scale=0.02)
    with oc.op_threads():
        x0 = oc.cgls_stat64(w, b, ang, maxit=2, tol=0.0)[0].astype(np.float32) if warm else None
        x64, t64 = oc.cgls_stat64(w, b, ang, maxit=4, tol=0.0, x0=x0)
        x_ref, t_ref = oc.cgls_stat(w, b, ang, maxit=4, tol=0.0, x0=x0)
    xd = vol_to_dev(plan, x0) if warm else empty_vol(plan)
    hist, info = plan.cgls_stat(sino_to_dev(plan, b), xd, 4, 0.0, warm=warm)
    assert info.iterations == 4
    close(vol_from_dev(plan, xd), hist, x64, t64.rel_history(), x_ref, t_ref.rel_history(), trace=not warm)
