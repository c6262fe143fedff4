"""Calls on one built handle at the same time, from host threads with streams of their own: each
gives what it gives alone."""
import threading

import pytest
import torch

import rtb200
from rtb200 import scenes

pytestmark = pytest.mark.gpu


def in_threads(n, work):
    failed = []

    def run(k):
        try:
            work(k)
        except BaseException as e:  # noqa: BLE001 - reported by the test's own thread
            failed.append((k, e))

    torch.cuda.synchronize()
    threads = [threading.Thread(target=run, args=(k,)) for k in range(n)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


@pytest.mark.parametrize("form", [-1, 2])
@pytest.mark.parametrize("n", [1000, 160001])
def test_traces(form, n):
    """Small batches and batches of more rays than the chip holds lanes, whose warps claim rays from a
    counter: every call's own rays are traced, each once."""
    v, t = scenes.soup(3000, seed=8, lo=1e-2, hi=1e-1)
    b = rtb200.Bvh.build(v, t, "lbvh63")
    b.trace_loop(form)
    rays = [torch.from_numpy(scenes.incoherent_rays(n, [0, 0, 0], [1, 1, 1], seed=k)).cuda() for k in range(8)]
    want = [b.trace(r) for r in rays]
    streams = [torch.cuda.Stream() for _ in rays]
    hits = [[torch.full_like(r, -7.0) for _ in range(4)] for r in rays]

    def work(k):
        for h in hits[k]:
            assert rtb200.lib().rt_trace(b.h, rays[k].data_ptr(), h.data_ptr(), n, 0, streams[k].cuda_stream) == 0

    in_threads(len(rays), work)
    for k, w in enumerate(want):
        assert all(torch.equal(h.view(torch.int32), w.view(torch.int32)) for h in hits[k]), k


def test_host_traces():
    """Rays from host memory: batches of different sizes, whose staging buffers grow on the way."""
    v, t = scenes.soup(3000, seed=8, lo=1e-2, hi=1e-1)
    b = rtb200.Bvh.build(v, t, "hybrid")
    rays = [scenes.incoherent_rays(1000 * 3 ** (k % 4) + k, [0, 0, 0], [1, 1, 1], seed=k) for k in range(12)]
    want = [rtb200.Bvh.build(v, t, "hybrid").trace(r) for r in rays]
    got = [[] for _ in rays]

    def work(k):
        for _ in range(3):
            got[k].append(b.trace(rays[k]))

    in_threads(len(rays), work)
    for k, w in enumerate(want):
        assert len(got[k]) == 3 and all(g.tobytes() == w.tobytes() for g in got[k]), k


def test_renders():
    """Images of different sizes and sample counts, whose scratch differs, some without any."""
    import numpy as np
    from test_gpu_paths import VIEW, scene
    b, mats, mot = scene("hybrid")
    dm, dmot = torch.from_numpy(rtb200.materials_array(mats)).cuda(), torch.from_numpy(mot.astype(np.int32)).cuda()
    cfgs = [rtb200.render_cfg(64 + 48 * k, 40 + 8 * k, 1 + k % 5, max_bounce=4, rr_after=1, env_kind=1, seed=k, lookat=VIEW)
            for k in range(8)]
    want = [b.render(c, dm, dmot, want_sq=True) for c in cfgs]
    got = [[] for _ in cfgs]

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            for i in range(6):
                got[k].append(b.render(cfgs[k], dm, dmot, mode=i % 2, want_sq=True))
            torch.cuda.current_stream().synchronize()

    in_threads(len(cfgs), work)
    for k, w in enumerate(want):
        assert len(got[k]) == 6 and all(torch.equal(g[0], w[0]) and torch.equal(g[1], w[1]) for g in got[k]), k
