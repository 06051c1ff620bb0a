"""The tensor-core projectors (square-pixel and Kaiser-Bessel plans of all but
small sizes) at the sizes where their blocks end: slice tiles of 128 and 256, 16 x
16-pixel tiles, angle groups and pairs, and with operands that the FP16 pairs
cannot hold.  References: the oracle with every sum in double.

TOL: both factors of a product carry 22 bits (2^-23 each, lo * lo 2^-24
dropped), a block's sum loses at most a few 2^-23 to rounding toward zero, the
sums over blocks are FP32: under 1e-6 for sums without cancellation, and
random-sign sums grow like their errors.  The Kaiser-Bessel weights are
interpolated in FP32: 1e-5, as for every kernel of that weighting.
"""
import numpy as np
import pytest

from conftest import rel_l2, uniform_angles
from devutil import empty_sino, empty_vol, sino_from_dev, sino_to_dev, vol_from_dev, vol_to_dev

pytestmark = pytest.mark.gpu

KB, SQ = 2, 3
TOL = {SQ: 1e-6, KB: 1e-5}


def make(gb, nx, ny, ang, w=SQ):
    plan = gb.Plan(w, 0.5 * (nx - 1), ny, np.asarray(ang, np.float32))
    assert plan.nx == nx
    return plan


def project(plan, x):
    qd = empty_sino(plan)
    qd.fill_(7.0)
    plan.project(vol_to_dev(plan, x), qd)
    return sino_from_dev(plan, qd)


def backproject(plan, s):
    gd = empty_vol(plan)
    gd.fill_(7.0)
    plan.backproject(sino_to_dev(plan, s), gd)
    return vol_from_dev(plan, gd)


ODD = np.concatenate([[1.475, 21.123, 2.123, -0.3, 7.9, 0.785398, 0.7853982, 2.3561945, 3.1415927],
                      uniform_angles(60)]).astype(np.float32)
FEW = [1e-4, 0.78, 0.79, 1.5707]
CASES = [
    (SQ, 32, 41, ODD), (SQ, 33, 49, ODD), (SQ, 32, 48, uniform_angles(65)),
    (SQ, 34, 120, uniform_angles(71)), (SQ, 48, 128, uniform_angles(72)),
    (SQ, 49, 129, uniform_angles(73)), (KB, 33, 136, uniform_angles(65)),
    (SQ, 65, 256, uniform_angles(64)), (SQ, 64, 257, uniform_angles(69, 2 * np.pi)),
    (KB, 65, 56, ODD), (SQ, 257, 44, uniform_angles(181)), (SQ, 530, 48, FEW), (SQ, 360, 41, [0.3]),
    (SQ, 32, 41, uniform_angles(4096)),  # the back projector's table of windows is full
    # few slices, taps computed by the kernels
    (SQ, 220, 1, ODD), (KB, 347, 8, ODD), (SQ, 1100, 20, FEW[:2]), (SQ, 96, 40, uniform_angles(250)),
]


@pytest.mark.parametrize("w,nx,ny,ang", CASES)
def test_edges(gb, oc, w, nx, ny, ang):
    plan = make(gb, nx, ny, ang, w)
    rng = np.random.default_rng(nx + ny)
    radius, ang = 0.5 * (nx - 1), np.asarray(ang, np.float32)
    x = rng.random((plan.nrays, ny), dtype=np.float32)
    s = rng.standard_normal((len(ang), ny, nx)).astype(np.float32)
    with oc.op_threads():
        q64, g64 = oc.project64(w, radius, x, ang), oc.backproject64(w, radius, s, ang)
    q, g = project(plan, x), backproject(plan, s)
    assert plan.check() == 0
    print("%s nx %d ny %d: forward %.1e, back %.1e" % (w, nx, ny, rel_l2(q, q64), rel_l2(g, g64)))
    assert rel_l2(q, q64) < TOL[w]
    assert rel_l2(g, g64) < TOL[w]


def test_constant_sinogram_keeps_its_sum(gb, oc):
    """Equal addends round the same way: 400 of them keep their sum."""
    nx, na = 48, 800
    plan = make(gb, nx, 41, uniform_angles(na))
    s = np.full((na, 41, nx), 8.517193, np.float32)
    with oc.op_threads():
        g64 = oc.backproject64(SQ, 0.5 * (nx - 1), s, uniform_angles(na))
    assert rel_l2(backproject(plan, s), g64) < 3e-7


@pytest.mark.parametrize("value", [1e6, -3.4028235e38, np.inf, -np.inf, np.nan])
def test_wide_values_stay_where_they_are(gb, oc, value):
    """One large or non-finite ray (or bin) of one slice: everything it does not
    reach is as without it, what it reaches is finite where the oracle's is."""
    nx, ny, ang = 65, 42, uniform_angles(64)
    plan = make(gb, nx, ny, ang)
    rng = np.random.default_rng(5)
    x = rng.random((plan.nrays, ny), dtype=np.float32)
    s = rng.random((len(ang), ny, nx), dtype=np.float32)
    ray, at = (plan.nrays // 3, 5), (11, 5, 30)
    clean = project(plan, x), backproject(plan, s)
    xu, su = np.zeros_like(x), np.zeros_like(s)
    xu[ray] = su[at] = 1.0
    touched = project(plan, xu) != 0, backproject(plan, su) != 0
    x[ray] = s[at] = value
    with oc.op_threads():
        ref = oc.project(SQ, 0.5 * (nx - 1), x, ang), oc.backproject(SQ, 0.5 * (nx - 1), s, ang)
    out2 = project(plan, x), backproject(plan, s)
    for out, c, hit, r in zip(out2, clean, touched, ref):
        far = ~hit & np.isfinite(r)
        np.testing.assert_allclose(out[far], c[far], rtol=2e-6, atol=2e-6 * np.abs(c).max())
        assert np.array_equal(np.isfinite(out), np.isfinite(r))
    assert plan.check() == 0


def test_streams_and_graphs_share_a_plan(gb):
    """Back and forward projections on two streams, and a captured pair replayed
    beside eager calls, give what they give alone."""
    import torch

    nx, ny, ang = 96, 44, uniform_angles(64)
    plan = make(gb, nx, ny, ang)
    rng = np.random.default_rng(9)
    n = 6
    vols = [vol_to_dev(plan, rng.random((plan.nrays, ny), dtype=np.float32)) for _ in range(n)]
    alone = []
    for v in vols:
        q, g = empty_sino(plan), empty_vol(plan)
        plan.project(v, q)
        plan.backproject(q, g)
        alone.append((q, g))
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = [(empty_sino(plan), empty_vol(plan)) for _ in vols]
    torch.cuda.synchronize()
    for rep in range(3):
        for i, v in enumerate(vols):
            st = streams[i % 2].cuda_stream
            plan.project(v, outs[i][0], stream=st)
            plan.backproject(outs[i][0], outs[i][1], stream=st)
    torch.cuda.synchronize()
    for a, o in zip(alone, outs):
        assert torch.equal(a[0], o[0]) and torch.equal(a[1], o[1])
    v, (q, g) = vols[0].clone(), (empty_sino(plan), empty_vol(plan))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=streams[0]):
        plan.project(v, q, stream=streams[0].cuda_stream)
        plan.backproject(q, g, stream=streams[0].cuda_stream)
    for i in range(n):
        torch.cuda.synchronize()
        v.copy_(vols[i])
        torch.cuda.synchronize()
        with torch.cuda.stream(streams[0]):
            graph.replay()
        for j in range(n):
            plan.project(vols[j], outs[j][0], stream=streams[1].cuda_stream)
            plan.backproject(outs[j][0], outs[j][1], stream=streams[1].cuda_stream)
        torch.cuda.synchronize()
        assert torch.equal(q, alone[i][0]) and torch.equal(g, alone[i][1])
        assert all(torch.equal(a[1], o[1]) for a, o in zip(alone, outs))


def test_cgls_is_no_further_from_fp64_than_the_reference(gb, oc):
    """Twelve steps at 48 slices: steps computed from <s, q> keep the directions
    conjugate whatever A and A^T lose to rounding."""
    w, nx, ny, its = SQ, 65, 48, 12
    ang, rng = uniform_angles(64), np.random.default_rng(31)
    plan = make(gb, nx, ny, ang)
    with oc.op_threads():
        b = oc.project(w, 0.5 * (nx - 1), rng.random((plan.nrays, ny), dtype=np.float32), ang)
        b = (b + 0.01 * rng.standard_normal(b.shape)).astype(np.float32)
        x64, _ = oc.cgls64(w, b, ang, maxit=its, tol=0.0)
        x_ref, _ = oc.cgls(w, b, ang, maxit=its, tol=0.0)
    xd = empty_vol(plan)
    plan.cgls(sino_to_dev(plan, b), xd, its, 0.0)
    e, e_ref = rel_l2(vol_from_dev(plan, xd), x64), rel_l2(x_ref, x64)
    print("cgls x%d: gpu-fp64 %.1e, ref-fp64 %.1e" % (its, e, e_ref))
    assert e < max(1e-5, 1.1 * e_ref)
