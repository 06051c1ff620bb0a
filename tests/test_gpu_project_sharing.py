"""Projections on two streams that share one plan, with and without FP64 norms, give
what they give alone: plans on the FP32 kernels (whose forward projection copies the
volume into column order first) and on the tensor cores."""
import pytest

from conftest import uniform_angles
from devutil import empty_sino, empty_vol

pytestmark = pytest.mark.gpu

# weighting, bins, angles, slices: FP32 with tables, tensor cores (CGLS not), tensor cores,
# linear weighting
PLANS = [(3, 200, 60, 48), (2, 96, 48, 40), (3, 230, 60, 40), (3, 128, 96, 64), (1, 96, 40, 24)]


@pytest.mark.parametrize("weighting,nx,na,ny", PLANS)
@pytest.mark.parametrize("norms", [False, True])
def test_two_streams(gb, weighting, nx, na, ny, norms):
    import torch

    plan = gb.Plan(weighting, 0.5 * (nx - 1), ny, uniform_angles(na))
    g = torch.Generator(device="cuda")
    g.manual_seed(nx)
    n = 6
    # scales of their own: a norm or a volume in the wrong place shows
    vols = [(i + 1) * torch.rand(plan.vol_shape, generator=g, device="cuda") for i in range(n)]

    def call(i, q, v, n2, stream):
        plan.project(vols[i], q, norm2=n2[0:1] if norms else None, stream=stream)
        plan.backproject(q, v, norm2=n2[1:2] if norms else None, stream=stream)

    def outputs():
        return empty_sino(plan), empty_vol(plan), torch.zeros(2, dtype=torch.float64, device="cuda")

    alone = [outputs() for _ in range(n)]
    for i in range(n):
        call(i, *alone[i], torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for rep in range(4):
        both = [outputs() for _ in range(n)]
        torch.cuda.synchronize()
        for i in range(n):
            call(i, *both[i], streams[(i + rep) % 2].cuda_stream)
        torch.cuda.synchronize()
        for a, b in zip(alone, both):
            assert all(torch.equal(x, y) for x, y in zip(a, b))
    assert plan.check() == 0
