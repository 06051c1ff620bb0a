"""What the tensor-core projectors give back for the tensor core's rounding toward zero
is the same share of every ray, wherever it lies: the mean scale of a row's projection
against the same row elsewhere in the image, over 1500 values and more.

Single values differ by their roundings (up to 2^-23, a bin's three rays may fall into
other blocks), their mean by 2^-23 / sqrt(1500) = 3e-9 at random and no more than that of
a few blocks: 2e-8.  A factor 1 + 2^-23 on the sums of some blocks and not of others
is 1.2e-7.
"""
import pytest

from conftest import uniform_angles
from devutil import empty_sino

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weighting,nx,ny", [(3, 257, 48), (3, 256, 136), (2, 257, 48)])
def test_scale_does_not_depend_on_the_place(gb, weighting, nx, ny):
    import torch

    plan = gb.Plan(weighting, 0.5 * (nx - 1), ny, uniform_angles(96))
    # rays row by row: the rows' first rays and pixels
    c = torch.arange(nx) - 0.5 * (nx - 1)
    t = torch.trunc(c).long() ** 2
    inside = t[:, None] + t[None, :] <= int((0.5 * (nx - 1)) ** 2)
    start, lo = torch.cumsum(inside.sum(1), 0) - inside.sum(1), inside.int().argmax(1)
    assert int(inside.sum()) == plan.nrays
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    w = nx // 4  # the middle columns: rays in all of the rows below
    row = torch.rand(w, plan.ys, generator=g, device="cuda") + 0.5
    sums = []
    for z in range(nx // 2 - 64, nx // 2 + 64, 8):
        x = torch.zeros(plan.vol_shape, device="cuda")
        k = int(start[z] + (nx - w) // 2 - lo[z])
        x[k:k + w] = row
        q = empty_sino(plan)
        plan.project(x, q)
        sums.append(float(q[0].double().sum()))  # angle 0: the row lies on its own bins
    spread = (max(sums) - min(sums)) / sums[0]
    print("weighting %d, nx %d: mean scale differs by %.1e" % (weighting, nx, spread))
    assert spread < 2e-8
