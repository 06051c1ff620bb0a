"""A graph of captured projections can be cloned, nested in another graph and
instantiated twice, on plans of the tensor-core projectors as on the others (graphs with
allocation nodes cannot), and its memory outlives the graph it was captured into."""
import ctypes

import pytest

from conftest import uniform_angles
from devutil import empty_sino, empty_vol

pytestmark = pytest.mark.gpu


def check(rc):
    assert rc == 0, "CUDA error %d" % rc


@pytest.mark.parametrize("nx,na,ny", [(96, 64, 56), (200, 64, 20), (65, 20, 12)])
def test_graphs_clone_nest_and_instantiate_twice(gb, nx, na, ny):
    import torch

    cu = ctypes.CDLL("libcuda.so.1")
    plan = gb.Plan(3, 0.5 * (nx - 1), ny, uniform_angles(na))
    g = torch.Generator(device="cuda")
    g.manual_seed(nx)
    vols = [torch.rand(plan.vol_shape, generator=g, device="cuda") for _ in range(4)]
    alone = []
    for v in vols:
        q, b = empty_sino(plan), empty_vol(plan)
        plan.project(v, q)
        plan.backproject(q, b)
        torch.cuda.synchronize()
        alone.append((q, b))
    x, q, b = vols[0].clone(), empty_sino(plan), empty_vol(plan)
    st = torch.cuda.Stream()
    s = ctypes.c_void_p(st.cuda_stream)
    torch.cuda.synchronize()
    base, clone, parent, node = (ctypes.c_void_p() for _ in range(4))
    check(cu.cuStreamBeginCapture_v2(s, 0))
    plan.project(x, q, stream=st.cuda_stream)
    plan.backproject(q, b, stream=st.cuda_stream)
    plan.project(x, q, stream=st.cuda_stream)  # shares the first one's memory
    check(cu.cuStreamEndCapture(s, ctypes.byref(base)))
    check(cu.cuGraphClone(ctypes.byref(clone), base))
    check(cu.cuGraphCreate(ctypes.byref(parent), 0))
    check(cu.cuGraphAddChildGraphNode(ctypes.byref(node), parent, None, ctypes.c_size_t(0), base))
    execs = []
    for gr in (base, base, clone, parent):
        e = ctypes.c_void_p()
        check(cu.cuGraphInstantiateWithFlags(ctypes.byref(e), gr, ctypes.c_ulonglong(0)))
        execs.append(e)
    check(cu.cuGraphDestroy(base))

    def replay(e, i):
        x.copy_(vols[i])
        q.zero_()
        b.zero_()
        torch.cuda.synchronize()
        check(cu.cuGraphLaunch(e, s))
        torch.cuda.synchronize()
        assert torch.equal(q, alone[i][0]) and torch.equal(b, alone[i][1])

    for i, e in enumerate(execs):
        replay(e, i)
    for e in execs[:3]:
        check(cu.cuGraphExecDestroy(e))
    check(cu.cuGraphDestroy(clone))
    other = gb.Plan(3, 0.5 * (nx - 1), ny, uniform_angles(na))  # frees what no graph holds
    replay(execs[3], 1)
    other.close()
    check(cu.cuGraphExecDestroy(execs[3]))
    check(cu.cuGraphDestroy(parent))
    plan.project(vols[2], q)
    torch.cuda.synchronize()
    assert torch.equal(q, alone[2][0])
    assert plan.check() == 0
    plan.close()
