"""Renders captured into CUDA graphs: kernels only, no memory of the graph's own, so that a caller may
instantiate the graph as often as it likes or use it as a child; bit-equal to the same call alone."""
import numpy as np
import pytest
import torch

import rtb200
from test_gpu_paths import VIEW, scene

pytestmark = pytest.mark.gpu


def device(mats, mot):
    return torch.from_numpy(rtb200.materials_array(mats)).cuda(), torch.from_numpy(mot.astype(np.int32)).cuda()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("w,h,spp", [(1, 1, 300), (7, 5, 3), (61, 43, 9), (700, 500, 2)])
def test_captured_render(mode, w, h, spp):
    from cuda.bindings import runtime as rt
    b, mats, mot = scene("hybrid")
    dm, dmot = device(mats, mot)
    rc = rtb200.render_cfg(w, h, spp, max_bounce=4, rr_after=1, env_kind=1, env_color=(0.1, 0.2, 0.3), seed=w, sample_offset=5,
                           lookat=VIEW)
    want = b.render(rc, dm, dmot, mode=mode, want_sq=True)
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        got = b.render(rc, dm, dmot, mode=mode, want_sq=True)
    raw = graph.raw_cuda_graph()
    _, _, count = rt.cudaGraphGetNodes(raw)
    _, nodes, _ = rt.cudaGraphGetNodes(raw, count)
    kinds = [rt.cudaGraphNodeGetType(n)[1] for n in nodes[:count]]
    assert set(kinds) == {rt.cudaGraphNodeType.cudaGraphNodeTypeKernel}, kinds
    execs = [rt.cudaGraphInstantiate(raw, 0) for _ in range(2)]
    for err, ex in execs:
        assert err == rt.cudaError_t.cudaSuccess
        for g in got:
            g.fill_(-1.0)
        torch.cuda.synchronize()
        assert rt.cudaGraphLaunch(ex, torch.cuda.current_stream().cuda_stream)[0] == rt.cudaError_t.cudaSuccess
        torch.cuda.synchronize()
        assert all(torch.equal(g, x) for g, x in zip(got, want))
    for _, ex in execs:
        rt.cudaGraphExecDestroy(ex)


def test_captured_batch_is_refused():
    """A render of several scenes uploads their cameras and cannot be captured: it says so and leaves
    the caller's graph as it was."""
    from cuda.bindings import runtime as rt
    from test_gpu_batch import batch_setup, cfgs_for
    scs, bb, mats, mot = batch_setup(n=3)
    dm, dmot = device(mats, mot)
    rcs = cfgs_for(scs, 32, 24, 2, max_bounce=3, rr_after=-1)
    want = bb.render_batch(rcs, dm, dmot)[0]
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    x = torch.zeros(8, device="cuda")
    with torch.cuda.graph(graph):
        x.add_(1.0)
        with pytest.raises(rtb200.RtError, match="RT_E_INVALID"):
            bb.render_batch(rcs, dm, dmot)
    assert rt.cudaGraphGetNodes(graph.raw_cuda_graph())[2] == 1
    assert torch.equal(bb.render_batch(rcs, dm, dmot)[0], want)
