"""The persistent path kernel where it can go wrong: images that are not whole tiles, fewer paths than
lanes, sample groups and launch pieces of every kind, calls on several streams, graph capture."""
import numpy as np
import pytest

import rtb200
from oracle import Baked
from render_checks import orc_cfg_from
from test_gpu_batch import batch_setup, cfgs_for
from test_gpu_render import compare, cornell_scene

pytestmark = pytest.mark.gpu
VIEW = ((0.0, 0.0, -2.9), (0.0, 0.0, 0.0), 45.0)


def scene(preset="lbvh30"):
    v, t, obj, mats = cornell_scene()
    b = rtb200.Bvh.build(v, t, preset)
    return b, mats, obj[b.prim_ids()]


@pytest.mark.parametrize("w,h,spp", [(1, 1, 300), (7, 5, 40), (8, 4, 33), (9, 33, 16), (61, 43, 9)])
def test_image_sizes_match_oracle(orc, w, h, spp):
    b, mats, mot = scene()
    nodes, tris, verts = b.download()
    rc = rtb200.render_cfg(w, h, spp, max_bounce=4, rr_after=1, env_kind=1, env_color=(0.1, 0.2, 0.3), seed=w, lookat=VIEW)
    rgb, rgb2 = b.render(rc, mats, mot, want_sq=True)
    ref, ref2 = orc.render(Baked(nodes, tris, verts), orc_cfg_from(rc), mats, mot, threads=8, want_sq=True)
    # a pixel sums spp samples; a sample differs where host and device cosf / sinf round apart
    compare(rgb, rgb2, ref, ref2, spp, f"{w}x{h}x{spp}", min_equal=0.0)


@pytest.mark.parametrize("chunk,stack,blk", [(1024, 64, 32), (4096, 64, 256), (16384, 64, 96), (1 << 26, 64, 128)])
def test_groups_and_pieces_give_the_same_image(chunk, stack, blk):
    """Samples are summed in order whatever the launches are: bit-equal images."""
    scs, bb, mats, mot = batch_setup(n=3)
    rcs = cfgs_for(scs, 50, 37, 7, max_bounce=4, rr_after=2)
    a, a2 = bb.render_batch(rcs, mats, mot, want_sq=True)
    c, c2 = bb.render_batch(rcs, mats, mot, params=rtb200.WavefrontParams(blk, chunk, stack, 256), want_sq=True)
    assert np.array_equal(a.cpu().numpy(), c.cpu().numpy()) and np.array_equal(a2.cpu().numpy(), c2.cpu().numpy())


def test_calls_on_two_streams():
    import torch
    b, mats, mot = scene("hybrid")
    rc = [rtb200.render_cfg(128, 96, 16, max_bounce=4, rr_after=-1, env_kind=1, seed=s, lookat=VIEW) for s in (1, 2)]
    want = [b.render(r, mats, mot)[0].cpu().numpy() for r in rc]
    streams = [torch.cuda.Stream() for _ in rc]
    dm, dmot = torch.from_numpy(rtb200.materials_array(mats)).cuda(), torch.from_numpy(mot.astype(np.int32)).cuda()
    torch.cuda.synchronize()
    got = []
    for k in range(6):
        with torch.cuda.stream(streams[k % 2]):
            got.append(b.render(rc[k % 2], dm, dmot)[0])
    torch.cuda.synchronize()
    for k, g in enumerate(got):
        assert np.array_equal(g.cpu().numpy(), want[k % 2]), k


def test_capture_and_replay():
    import torch
    b, mats, mot = scene("hybrid")
    rc = rtb200.render_cfg(40, 30, 8, max_bounce=4, rr_after=-1, env_kind=1, seed=3, lookat=VIEW)
    dm, dmot = torch.from_numpy(rtb200.materials_array(mats)).cuda(), torch.from_numpy(mot.astype(np.int32)).cuda()
    alb = torch.rand(mot.shape[0], 3, device="cuda")
    want = b.render(rc, dm, dmot, tri_albedo=alb)[0].cpu().numpy()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        img = b.render(rc, dm, dmot, tri_albedo=alb)[0]
    graph.replay()
    assert np.array_equal(img.cpu().numpy(), want)
    alb.mul_(0.5)
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(img.cpu().numpy(), b.render(rc, dm, dmot, tri_albedo=alb)[0].cpu().numpy())


def test_adjoint_does_not_depend_on_zero_pixels():
    """Pixels with dLoss/dI = 0 are skipped: the gradients of the others are those of their paths alone."""
    import torch
    b, mats, mot = scene()
    rc = rtb200.render_cfg(33, 21, 12, max_bounce=4, rr_after=2, env_kind=1, seed=5, lookat=VIEW)
    d = torch.zeros(21, 33, 3, device="cuda")
    d[:, ::3] = 1.0
    rest = torch.ones_like(d) - d
    one, two, full = (b.adjoint(rc, x, mats, mot) for x in (d, rest, torch.ones_like(d)))
    for k in range(2):
        total = (one[k].double() + two[k].double()).cpu().numpy()
        ref = full[k].double().cpu().numpy()
        # float sums of the same terms in other orders
        assert np.linalg.norm(total - ref) <= 1e-4 * np.linalg.norm(ref)


def test_short_albedo_table():
    """A table with fewer rows than baked triangles: the missing rows are black."""
    import torch
    b, mats, mot = scene()
    rc = rtb200.render_cfg(24, 16, 4, max_bounce=3, rr_after=-1, env_kind=1, seed=2, lookat=VIEW)
    n = mot.shape[0]
    full = torch.full((n, 3), 0.5)
    full[n // 2:] = 0.0
    a = b.render(rc, mats, mot, tri_albedo=full)[0]
    c = b.render(rc, mats, mot, tri_albedo=full[:n // 2])[0]
    assert torch.equal(a, c)


@pytest.mark.parametrize("w,h", [(1, 1), (8, 4), (61, 43), (256, 256)])
def test_one_sample_of_a_small_image(w, h):
    """One launch, and the sample that an image of two samples has."""
    import torch
    b, mats, mot = scene("hybrid")
    dm, dmot = torch.from_numpy(rtb200.materials_array(mats)).cuda(), torch.from_numpy(mot.astype(np.int32)).cuda()

    def render(spp, offset):
        rc = rtb200.render_cfg(w, h, spp, max_bounce=4, rr_after=1, env_kind=1, env_color=(0.1, 0.2, 0.3), seed=w, sample_offset=offset,
                               lookat=VIEW)
        n = rtb200.lib().rt_kernel_launches()
        out = b.render(rc, dm, dmot, want_sq=True)
        return out, rtb200.lib().rt_kernel_launches() - n

    (x, x2), n0 = render(1, 3)
    (y, y2), n1 = render(1, 4)
    (z, z2), _ = render(2, 3)
    assert (n0, n1) == (1, 1)
    assert torch.equal((x + y) / 2, z) and torch.equal((x2 + y2) / 2, z2)


def test_tensors_made_for_a_call_on_another_stream():
    """The rest of a short albedo table and the gradients' zeros are made on the current stream, which
    is busy, and used on the call's; their memory is not handed out again while that one works."""
    import torch
    b, mats, mot = scene()
    rc = rtb200.render_cfg(64, 48, 64, max_bounce=4, rr_after=-1, env_kind=1, env_color=(0.4, 0.5, 0.6), seed=2, lookat=VIEW)
    n = mot.shape[0]
    mats, mot = torch.from_numpy(rtb200.materials_array(mats)).cuda(), torch.from_numpy(mot.astype(np.int32)).cuda()
    alb = torch.rand(n // 2, 3, device="cuda")
    d = torch.ones(48, 64, 3, device="cuda")
    want = b.render(rc, mats, mot, tri_albedo=alb)[0]
    grad = b.adjoint(rc, d, mats, mot, tri_albedo=alb)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    torch.cuda._sleep(1 << 28)  # the current stream is busy for about 0.15 s
    got = b.render(rc, mats, mot, tri_albedo=alb, stream=side)[0]
    fill = [torch.full((n, 3), 7.0, device="cuda") for _ in range(8)]
    g = b.adjoint(rc, d, mats, mot, tri_albedo=alb, stream=side.cuda_stream)
    fill += [torch.full((n, 3), 7.0, device="cuda") for _ in range(8)]
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    for x, y in zip(g, grad):  # float sums of the same terms in other orders
        assert float((x.double() - y.double()).norm()) <= 1e-4 * float(y.double().norm())


@pytest.mark.parametrize("w,h", [(1, 33), (3, 70), (7, 4), (33, 1), (100, 3), (9, 5)])
def test_narrow_and_low_images_match_oracle(orc, w, h):
    b, mats, mot = scene()
    rc = rtb200.render_cfg(w, h, 8, max_bounce=3, rr_after=1, env_kind=1, env_color=(0.1, 0.2, 0.3), seed=w, lookat=VIEW)
    rgb, rgb2 = b.render(rc, mats, mot, want_sq=True)
    ref, ref2 = orc.render(Baked(*b.download()), orc_cfg_from(rc), mats, mot, threads=8, want_sq=True)
    compare(rgb, rgb2, ref, ref2, 8, f"{w}x{h}", min_equal=0.0)


@pytest.mark.parametrize("w,h", [(1, 600_000_000), (1_200_000_000, 1)])
def test_long_thin_images(w, h):
    """Every pixel of an image far longer than wide is rendered: the background, with the scene behind the
    camera."""
    import torch
    b, _, _ = scene()
    rc = rtb200.render_cfg(w, h, 1, max_bounce=1, rr_after=-1, env_kind=1, env_color=(0.25, 0.5, 0.75), seed=1,
                           lookat=((0.0, 0.0, -9.0), (0.0, 0.0, -10.0), 45.0))
    img = b.render(rc)[0].reshape(-1, 3)
    for c in range(3):
        assert torch.aminmax(img[:, c]) == (0.25 * (c + 1), 0.25 * (c + 1))
    del img
    torch.cuda.empty_cache()
