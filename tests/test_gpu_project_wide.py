"""Operands whose slices span more than the tensor-core projectors' FP16 pairs hold:
a few large finite values beside ordinary or small ones.  References: the oracle with
every sum in double.

TOL: the rays and bins that the large values do not reach keep FP32's precision: sums
of at most 200 positive products, each rounded by 2^-24, and the weights' own rounding,
under 1e-6 (the pairs alone lose 2^-51 of the largest value: from 3e-6 of the sums at a
span of 1e11 on).
"""
import numpy as np
import pytest

from conftest import rel_l2, uniform_angles
from devutil import empty_sino, empty_vol, sino_from_dev, sino_to_dev, vol_from_dev, vol_to_dev

pytestmark = pytest.mark.gpu

KB, SQ = 2, 3
TOL = {SQ: 1e-6, KB: 1e-5}

# weighting, bins, slices, the slice that holds the large values
SHAPES = [(SQ, 65, 42, 41), (SQ, 33, 130, 0), (KB, 65, 264, 263), (SQ, 160, 9, 8), (SQ, 32, 4104, 4103)]


def operand(rng, shape, axis, y, scale, value, at):
    """Values of about `scale`; slice y (along `axis`) holds `value` at `at`."""
    v = (rng.random(shape, dtype=np.float32) + np.float32(0.5)) * np.float32(scale)
    np.moveaxis(v, axis, 0)[(y,) + at] = value
    return v


@pytest.mark.parametrize("w,nx,ny,y", SHAPES)
@pytest.mark.parametrize("scale,value", [(1.0, 1e9), (1.0, 1e10), (1.0, 1e11), (1.0, -1e12),
                                         (0.01, 1e9), (0.01, 1e12), (1e-20, 1.0)])
def test_large_values_leave_the_rest_exact(gb, oc, w, nx, ny, y, scale, value):
    na = 64 if ny > 9 else 100
    radius, ang = 0.5 * (nx - 1), uniform_angles(na)
    plan = gb.Plan(w, radius, ny, ang)
    rng = np.random.default_rng(nx + ny)
    ray, bin_ = (plan.nrays // 3,), (na // 5, nx // 2)
    x = operand(rng, (plan.nrays, ny), 1, y, scale, value, ray)
    s = operand(rng, (na, ny, nx), 1, y, scale, value, bin_)
    xu, su = np.zeros((plan.nrays, 1), np.float32), np.zeros((na, 1, nx), np.float32)
    xu[ray], su[bin_[0], 0, bin_[1]] = 1.0, 1.0
    with oc.op_threads():
        q64, g64 = oc.project64(w, radius, x, ang), oc.backproject64(w, radius, s, ang)
        hit_q = oc.project64(w, radius, xu, ang)[:, 0] != 0
        hit_g = oc.backproject64(w, radius, su, ang)[:, 0] != 0
    qd, gd = empty_sino(plan), empty_vol(plan)
    plan.project(vol_to_dev(plan, x), qd)
    plan.backproject(sino_to_dev(plan, s), gd)
    q, g = sino_from_dev(plan, qd)[:, y], vol_from_dev(plan, gd)[:, y]
    e_q, e_g = rel_l2(q[~hit_q], q64[:, y][~hit_q]), rel_l2(g[~hit_g], g64[:, y][~hit_g])
    print("%g beside %g: forward %.1e, back %.1e" % (value, scale, e_q, e_g))
    assert plan.check() == 0
    assert e_q < TOL[w] and e_g < TOL[w]
    assert rel_l2(q[hit_q], q64[:, y][hit_q]) < TOL[w] and rel_l2(g[hit_g], g64[:, y][hit_g]) < TOL[w]


@pytest.mark.parametrize("nx,ny", [(65, 48), (65, 131), (130, 256)])
def test_ordinary_slices_do_not_count_as_wide(gb, nx, ny):
    """Values around zero (some far below 2^-30 of the largest) and slices of zeros
    with a few values stay on the tensor cores: a scaled copy beside one that spans
    too much gives other last places than alone, an ordinary one the same."""
    import torch

    plan = gb.Plan(SQ, 0.5 * (nx - 1), ny, uniform_angles(64))
    g = torch.Generator(device="cuda")
    g.manual_seed(nx)
    x = torch.randn(plan.vol_shape, generator=g, device="cuda")
    x[:, 3] = 0.0
    x[plan.nrays // 2, 3] = 1.0
    x[7, 5] *= 2.0 ** -60
    alone, beside, wide = (empty_sino(plan) for _ in range(3))
    plan.project(x[:, :].clone(), alone)
    y = x.clone()
    y[:, 0] *= 4.0
    plan.project(y, beside)
    assert torch.equal(alone[:, :, 1:], beside[:, :, 1:])
    y[:, 0] = 1e-12
    y[0, 0] = 1.0  # one slice beyond the pairs: the whole operand leaves them
    plan.project(y, wide)
    assert not torch.equal(alone[:, :, 1:], wide[:, :, 1:])
    torch.testing.assert_close(wide[:, :, 1:], alone[:, :, 1:], rtol=0, atol=1e-4)


@pytest.mark.parametrize("value", [1e12, float("inf"), float("nan")])
def test_one_bad_value_costs_no_more_than_fp32(gb, value):
    """A dead pixel in one slice: the FP32 kernels take 2.4 to 4.8 times the tensor-core
    ones' time at these sizes, half as much again without the plan's tables."""
    import torch

    nx, na, ny = 256, 180, 64
    plan = gb.Plan(SQ, 0.5 * (nx - 1), ny, uniform_angles(na))
    x = torch.rand(plan.vol_shape, device="cuda")
    s = torch.rand(plan.sino_shape, device="cuda")
    q, g = empty_sino(plan), empty_vol(plan)

    def best(f):
        t = []
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            f(stream=torch.cuda.current_stream().cuda_stream)
            b.record()
            torch.cuda.synchronize()
            t.append(a.elapsed_time(b))
        return min(t)

    def forward(stream):
        plan.project(x, q, stream=stream)

    def back(stream):
        plan.backproject(s, g, stream=stream)

    clean = best(forward), best(back)
    x[plan.nrays // 2, 7] = s[na // 2, nx // 2, 7] = value
    bad = best(forward), best(back)
    print("%g: forward %.2f -> %.2f ms, back %.2f -> %.2f ms" % (value, clean[0], bad[0], clean[1], bad[1]))
    assert bad[0] < 8 * clean[0] and bad[1] < 8 * clean[1]
