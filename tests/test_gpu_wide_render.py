"""Wavefront and batched renders of a handle in form 2 trace its 8-wide layout, plain ones the binary
tree. Seen on pairs of coincident triangles of different emission, where the two visiting orders report
different triangles: a pixel of one sample is red or green by the triangle found first."""
import numpy as np
import pytest
import torch

import rtb200
from rtb200 import scenes

pytestmark = pytest.mark.gpu
VIEW = ((0.5, 0.5, -1.4), (0.5, 0.5, 0.5), 45.0)


def pairs(seed):
    v, t = scenes.soup(400, seed=seed, lo=5e-2, hi=2e-1)
    return v, np.repeat(t, 2, axis=0)


MATS = [dict(albedo=(0.0,) * 3, emission=(1.0, 0.0, 0.0)), dict(albedo=(0.0,) * 3, emission=(0.0, 1.0, 0.0))]


def check(binary, wide):
    a, c = binary.cpu().numpy(), wide.cpu().numpy()
    assert a.max() == 1.0
    assert np.array_equal(a[..., 0] + a[..., 1], c[..., 0] + c[..., 1])  # the same rays hit
    assert np.any(a != c)                                              # but not the same triangles


def test_single_scene():
    v, t = pairs(3)
    b = rtb200.Bvh.build(v, t, rtb200.make_cfg("lbvh63", max_leaf=1))
    mot = (b.prim_ids() % 2).astype(np.uint32)
    rc = rtb200.render_cfg(96, 80, 1, max_bounce=0, rr_after=-1, env_kind=1, seed=3, lookat=VIEW)
    rays = scenes.incoherent_rays(20000, [0, 0, 0], [1, 1, 1], seed=4)
    first = b.trace(rays)
    plain, wave = (b.render(rc, MATS, mot, mode=m)[0] for m in (0, 1))
    assert torch.equal(plain, wave)
    b.trace_loop(2)
    second = b.trace(rays)
    assert np.array_equal(first["t"], second["t"]) and np.any(first["tri"] != second["tri"])
    assert torch.equal(b.render(rc, MATS, mot, mode=0)[0], plain)
    wide = b.render(rc, MATS, mot, mode=1)[0]
    check(plain, wide)
    graph = torch.cuda.CUDAGraph()
    dm, dmot = torch.from_numpy(rtb200.materials_array(MATS)).cuda(), torch.from_numpy(mot.astype(np.int32)).cuda()
    with torch.cuda.graph(graph):
        got = b.render(rc, dm, dmot, mode=1)[0]
    graph.replay()
    assert torch.equal(got, wide)


@pytest.mark.parametrize("stack", [32, 64])
def test_batch(stack):
    parts = [pairs(5), pairs(6)]
    v, t, vo, to = rtb200.batch_arrays(parts)
    b = rtb200.Bvh.build_batch(v, t, vo, to, rtb200.make_cfg("lbvh30", max_leaf=1))
    assert b.depth() < 31
    mot = (b.prim_ids() % 2).astype(np.uint32)
    rcs = [rtb200.render_cfg(96, 80, 1, max_bounce=0, rr_after=-1, env_kind=1, seed=s, lookat=VIEW) for s in (1, 2)]
    params = rtb200.WavefrontParams(128, 1 << 20, stack, 256)
    binary = b.render_batch(rcs, MATS, mot, params=params)[0]
    b.trace_loop(2)
    wide = b.render_batch(rcs, MATS, mot, params=params)[0]
    for s in range(2):
        check(binary[s], wide[s])
