"""The warp-cooperative trace kernel at the sizes and inputs where it can go wrong: ray counts around
a warp and below one ray per resident warp, leaves of one to hundreds of triangles, rays and
vertices that are not finite. Bar: bit-equal to the oracle's restatement of bvh::trace."""
import numpy as np
import pytest
import torch

import rtb200
from oracle import Baked
from rtb200 import scenes
from test_gpu_trace import compare, rays_for

pytestmark = pytest.mark.gpu


def build(kind, preset, **kw):
    if kind == "soup":
        v, t = scenes.soup(3001, seed=5, lo=1e-2, hi=2e-1)
    else:  # runs of equal triangles: leaves far above 32 pairs
        v, t = scenes.soup(40, seed=6, lo=1e-1, hi=3e-1)
        t = np.repeat(t, 37, axis=0)
    return v, t, rtb200.Bvh.build(v, t, rtb200.make_cfg(preset, **kw))


@pytest.mark.parametrize("kind,preset,kw", [("soup", "lbvh63", {}), ("soup", "sah4", {}), ("soup", "lbvh63", dict(max_leaf=200)),
                                            ("soup", "lbvh63", dict(max_leaf=1)), ("runs", "lbvh63", dict(max_leaf=500)),
                                            ("runs", "hybrid", {})])
@pytest.mark.parametrize("flags", [0, 1, 2, 3])
def test_leaf_sizes(orc, kind, preset, kw, flags):
    v, t, b = build(kind, preset, **kw)
    nodes, tris, verts = b.download()
    rays = rays_for(v, 6001, seed=11)
    compare(b.trace(rays, flags), orc.trace(Baked(nodes, tris, verts), rays, flags=flags, threads=8), f"{kind}/{preset}/{kw}/{flags}")


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 1000, 4735, 4737, 151551, 151553])
def test_ray_counts(orc, n):
    v, t, b = build("soup", "hybrid")
    nodes, tris, verts = b.download()
    rays = rays_for(v, max(n, 8), seed=n)[:n]
    compare(b.trace(rays), orc.trace(Baked(nodes, tris, verts), rays, threads=8), f"n={n}")


@pytest.mark.parametrize("flags", [0, 1])
def test_rays_that_are_not_finite(orc, flags):
    v, t, b = build("soup", "lbvh63")
    nodes, tris, verts = b.download()
    rays = rays_for(v, 8192, seed=3)
    rng = np.random.default_rng(4)
    bad = np.array([np.nan, np.inf, -np.inf, 0.0, -0.0, 1e-45, -1e-45, 3e38, -3e38], np.float32)
    at = rng.integers(0, 8, 4096)
    rays[np.arange(4096), at] = bad[rng.integers(0, len(bad), 4096)]
    hits = b.trace(rays, flags)
    h, out, tri, counters, overflow = orc.trace(Baked(nodes, tris, verts), rays, flags=flags, threads=8)
    # x86 and CUDA give a NaN different sign bits: a NaN weight equals any NaN
    got = np.stack([hits["t"], hits["u"], hits["v"], hits["n"][:, 0], hits["n"][:, 1], hits["n"][:, 2]], axis=1)
    both = np.isnan(got) & np.isnan(out)
    out = np.where(both, got, out)
    compare(hits, (h, out, tri, counters, overflow), f"flags {flags}")


@pytest.mark.parametrize("preset", ["lbvh63", "hybrid"])
def test_vertices_that_are_not_finite(orc, preset):
    v, t = scenes.soup(600, seed=8, lo=1e-2, hi=2e-1)
    rng = np.random.default_rng(9)
    v[rng.integers(0, v.shape[0], 6), rng.integers(0, 3, 6)] = np.nan
    b = rtb200.Bvh.build(v, t, preset)
    nodes, tris, verts = b.download()
    rays = rays_for(np.nan_to_num(v), 8192, seed=10)
    compare(b.trace(rays), orc.trace(Baked(nodes, tris, verts), rays, threads=8), preset)


def test_traces_from_several_threads():
    """More calls at a time than there are status words, on streams of their own."""
    import threading
    v, t = scenes.soup(3000, seed=8, lo=1e-2, hi=1e-1)
    b = rtb200.Bvh.build(v, t, "hybrid")
    rays = torch.from_numpy(scenes.incoherent_rays(777, [0, 0, 0], [1, 1, 1], seed=4)).cuda()
    want, got = b.trace(rays).cpu(), [None] * 80

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(3):
                h = b.trace(rays)
            got[k] = h.cpu()

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(got))]
    for x in threads:
        x.start()
    for x in threads:
        x.join()
    assert all(g is not None and torch.equal(g.view(torch.int32), want.view(torch.int32)) for g in got)


@pytest.mark.parametrize("n", [1, 700, 160000])
def test_stack_overflow_is_reported(n):
    """A chain deeper than the 64-entry stack: the call reports it (code 5), and only that call."""
    depth = 80
    nodes = np.zeros(2 * depth + 1, rtb200.NODE_DTYPE)
    nodes["bmin"][:, :3], nodes["bmax"][:, :3] = 0.0, 1.0
    for i in range(depth):  # inner nodes 0 .. depth - 1, each with the next one and a leaf in an equal box
        nodes["a"][i], nodes["b"][i] = i + 1, 2 * depth - i
    nodes["is_leaf"][depth:] = 1
    nodes["b"][depth:] = 1
    verts = np.zeros((3, 6), np.float32)
    verts[:, :3] = [[0, 0, 0.5], [0, 1, 0.5], [1, 0, 0.5]]
    verts[:, 5] = 1.0
    b = rtb200.Bvh.from_arrays(nodes, np.array([[0, 1, 2]], np.uint32), verts)
    rays = torch.zeros(n, 8, device="cuda")
    rays[:, 0:3] = torch.tensor([0.2, 0.2, -1.0])
    rays[:, 6], rays[:, 7] = 1.0, float("inf")
    off = rays.clone()
    off[:, 0] = 9.0
    hits = torch.empty_like(rays)

    def call(r):
        torch.cuda.synchronize()
        return rtb200.lib().rt_trace(b.h, r.data_ptr(), hits.data_ptr(), n, 0, None)

    assert [call(rays), call(off), call(rays), call(off)] == [5, 0, 5, 0]


def test_axis_parallel_rays_cost_what_others_do():
    """Orthographic rays (two direction components 0) take the general box test at every node, with the
    reciprocals of the ray's start: the same grid tilted a little takes the same nodes without it. 1.11-1.12 times
    the time on a B200; 1.40 while the reciprocals were taken again at every node."""
    v, t = scenes.icosphere(6, seed=2)
    b = rtb200.Bvh.build(v, t, "sah4")
    n = 1024
    y, x = torch.meshgrid(torch.linspace(-1, 1, n, device="cuda"), torch.linspace(-1, 1, n, device="cuda"), indexing="ij")
    rays = torch.zeros(n * n, 8, device="cuda")
    rays[:, 0], rays[:, 1], rays[:, 2], rays[:, 6], rays[:, 7] = x.reshape(-1), y.reshape(-1), -2.0, 1.0, float("inf")
    tilted = rays.clone()
    tilted[:, 4], tilted[:, 5] = 1e-3, 2e-3
    hits = torch.empty_like(rays)

    def once(r):
        a, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        assert rtb200.lib().rt_trace(b.h, r.data_ptr(), hits.data_ptr(), n * n, 0, 1) == 0  # (torch's default stream)
        e.record()
        e.synchronize()
        return a.elapsed_time(e)

    times = np.array([[once(rays), once(tilted)] for _ in range(24)])[4:]
    assert np.median(times[:, 0] / times[:, 1]) < 1.2, times


def test_long_rays_among_others():
    """The cap on a ray's steps counts its own nodes only. A few rays with 32,768 leaves share a warp with
    rays of eight million nodes, for which they wait at every leaf: 2^24 rounds of the warp in all, and no
    ray near the cap of 2^24. (The tree is a DAG: chains of nodes whose children are the next one.)"""
    far = np.array([[100.0, 0, 0], [101.0, 1, 1]])

    def box(x0, x1, z0, z1):
        return np.array([[x0, 0.0, z0], [x1, 1.0, z1]])

    recs = [[box(0, 3, 0, 3), 0, 0, 0], [box(1, 3, 0, 3), 0, 0, 0], [box(2, 3, 0, 3), 0, 0, 0]]

    def chain(depth, b, leaf_box):  # `depth` inner nodes, the last with two equal leaves: 2^depth - 1 visits
        first = len(recs)
        recs.extend([b, 0, first + k + 1, first + k + 1] for k in range(depth))
        recs.append([leaf_box, 1, 0, 1])
        return first

    near, deep = 15, 23
    recs[0][2:] = [chain(near, box(0, 1, 0, 1), box(0, 1, 0, 1)), 1]
    recs[1][2:] = [chain(deep, box(1, 2, 2, 3), far), 2]
    recs[2][2:] = [chain(near - 1, box(2, 3, 0, 1), box(2, 3, 0, 1)), chain(deep, box(2, 3, 2, 3), far)]
    nodes = np.zeros(len(recs), rtb200.NODE_DTYPE)
    for i, (b, leaf, left, right) in enumerate(recs):
        nodes["bmin"][i, :3], nodes["bmax"][i, :3] = b
        nodes["is_leaf"][i], nodes["a"][i], nodes["b"][i] = leaf, left, right
    verts = np.zeros((3, 6), np.float32)  # no area: every leaf is tested, none is hit
    b = rtb200.Bvh.from_arrays(nodes, np.array([[0, 1, 2]], np.uint32), verts)
    n = 151552  # a ray for each resident lane, by index: the first warp has the first 32
    rays = torch.zeros(n, 8, device="cuda")
    rays[:, 0], rays[:, 1], rays[:, 2], rays[:, 7] = 9.0, 0.5, -1.0, float("inf")
    rays[:, 4], rays[:, 5], rays[:, 6] = 1e-3, 1e-3, 1.0
    rays[:4, 0], rays[4:18, 0], rays[18:32, 0] = 0.5, 1.5, 2.5
    hits = torch.full_like(rays, -1.0)
    torch.cuda.synchronize()
    assert rtb200.lib().rt_trace(b.h, rays.data_ptr(), hits.data_ptr(), n, 0, None) == 0, rtb200.lib().rt_last_error()
    assert int(hits.view(torch.int32)[:, 7].abs().max()) == 0
