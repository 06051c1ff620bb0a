"""With little device memory left, what the library keeps for speed is no reason for a call
to fail: a plan does without the tensor-core projectors' FP16 operands rather than take
the room of a solve that fits beside it, and scratch kept between calls is given back."""
import pytest

from conftest import rel_l2, uniform_angles

pytestmark = pytest.mark.gpu


def test_a_solve_still_fits_beside_the_plan(gb):
    import torch

    nx, na, ny = 512, 400, 256
    ang = uniform_angles(na)
    big = gb.Plan(3, 0.5 * (nx - 1), ny, ang)
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    b = torch.zeros(big.sino_shape, device="cuda")
    big.project(torch.rand(big.vol_shape, generator=g, device="cuda"), b)
    x, want = torch.zeros(big.vol_shape, device="cuda"), torch.zeros(big.vol_shape, device="cuda")
    big.cgls(b, want, 3, 0.0)
    big.close()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    # operands 478 MB, under 40 % of what is left; CGLS's workspace 1.05 GB
    free, _ = torch.cuda.mem_get_info()
    left = 1300 << 20
    fill = torch.empty(free - left, dtype=torch.uint8, device="cuda")
    try:
        plan = gb.Plan(3, 0.5 * (nx - 1), ny, ang)
        plan.cgls(b, x, 3, 0.0)
        assert plan.check() == 0
        plan.close()
    finally:
        del fill
        torch.cuda.empty_cache()
    # the FP32 kernels against the tensor cores: rounding over three steps
    assert rel_l2(x.cpu().numpy(), want.cpu().numpy()) < 1e-5


def test_kept_scratch_is_given_back(gb):
    """After a shift search (252 MB of scratch, kept) a solve needs 253 MB of the 400 MB
    that were left before it."""
    import torch

    plan = gb.Plan(1, 127.5, 256, uniform_angles(180))
    b, x = torch.ones(plan.sino_shape, device="cuda"), torch.zeros(plan.vol_shape, device="cuda")
    a = torch.rand(5, 2048, 2048, device="cuda")
    sx, sy = torch.zeros(5, device="cuda"), torch.zeros(5, device="cuda")
    gb.cc_shifts(a, a, sx, sy)
    torch.cuda.synchronize()
    gb.Plan(1, 8.0, 8, uniform_angles(4)).close()  # gives the scratch back
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    fill = torch.empty(free - (400 << 20), dtype=torch.uint8, device="cuda")
    try:
        gb.cc_shifts(a, a, sx, sy)
        _, info = plan.cgls(b, x, 2, 0.0)
        assert info.iterations == 2
        assert float(sx.abs().max()) < 1e-3 and plan.check() == 0
        plan.close()
    finally:
        del fill
        torch.cuda.empty_cache()
