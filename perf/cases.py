"""Performance cases: what a program that uses this library has it do.

Each case is one pass through the public entry points (``rtb200.Bvh`` and the C ABI behind it):
baking a mesh (host arrays to host arrays, or device arrays into a handle), tracing ray
batches, path-traced images (per-pixel and wavefront schedule), a batch of scenes baked and
rendered together, and one step of differentiable rendering. Sizes are those of the repository's
benchmark configurations and tests; ``draw`` gives other sizes, presets, scenes and options of
the same ranges. Geometry is generated on the GPU from the seed.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("ray-tracer_b200"))

import rtb200  # noqa: E402

INF = float("inf")
LEAF = {"hybrid": 8.0, "lbvh63": 9.0, "lbvh30": 9.0, "sah4": 2.0, "sah16": 8.0}  # triangles per leaf, roughly


# ---- the cases ---------------------------------------------------------------------------------

def listed():
    return [
        # A prop or a collision proxy baked from host arrays, the baked arrays taken back to be written
        # to a file (what bvh::bakeBVH does), with the reference's own settings. The smallest call.
        dict(name="bake_host_5k", kind="bake_host", scene="mesh", n=5120, preset="hybrid", pinned=False),
        # The same for a scanned mesh, in pinned buffers, as an asset pipeline streams them.
        dict(name="bake_host_300k", kind="bake_host", scene="mesh", n=300007, preset="hybrid", pinned=True),
        # The headline build: a deforming mesh re-baked on the device every frame.
        dict(name="bake_lbvh63_1m", kind="bake", scene="soup", n=1048576, preset="lbvh63"),
        # The largest build.
        dict(name="bake_lbvh63_16m", kind="bake", scene="soup", n=16777216, preset="lbvh63"),
        # A high-quality tree for a static scene: binned SAH with spatial splits, leaves of 4.
        dict(name="bake_sah4_1m", kind="bake", scene="soup", n=1048576, preset="sah4"),
        # A handful of rays against a small mesh: picking, line of sight.
        dict(name="trace_small", kind="trace", scene="mesh", n=5120, preset="hybrid", rays="inside", n_rays=1000, flags=0),
        # One camera's visibility and its shadow rays at full HD against a large scene in the
        # reference's default tree: coherent closest hits, then any-hit rays towards a light.
        dict(name="camera_shadow_1080p", kind="camera", scene="spheres", n=1000003, preset="hybrid", width=1920, height=1080),
        # The microbenchmark's incoherent rays: bounced light, ambient occlusion, sampling queries.
        dict(name="trace_incoherent_4m", kind="trace", scene="soup", n=1048576, preset="lbvh63", rays="inside",
             n_rays=4194304, flags=0),
        # A small path-traced image with the default schedule (one thread per pixel).
        dict(name="render_plain_256", kind="render", scene="cornell", n=20480, preset="lbvh30", width=256, height=256, spp=16,
             max_bounce=4, rr_after=-1, wavefront=False),
        # The large image: five million triangles, mirrors, roulette, the wavefront schedule.
        dict(name="render_wavefront_1080p", kind="render", scene="spheres", n=5000000, preset="sah4", width=1920, height=1080,
             spp=64, max_bounce=8, rr_after=2, wavefront=True),
        # A data set's worth of scenes of uneven sizes, baked in one call and rendered in one call.
        dict(name="batch_64_scenes", kind="batch", n_scenes=64, lo=1000, hi=500000, width=512, height=512, spp=4, max_bounce=5,
             preset="lbvh30"),
        # One step of inverse rendering: the image (forward) and the gradients of per-triangle albedo
        # and emission (backward).
        dict(name="diff_step_512", kind="diff", n=50000, preset="lbvh30", width=512, height=512, spp=32, max_bounce=4),
    ]


def _log_int(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["bake_host", "bake", "trace", "trace", "camera", "render", "render", "batch", "diff"])
    if kind == "bake_host":
        return dict(kind=kind, scene=rng.choice(["mesh", "soup"]), n=_log_int(rng, 500, 500000),
                    preset=rng.choice(["hybrid", "lbvh63", "sah16"]), pinned=rng.random() < 0.5)
    if kind == "bake":
        preset = rng.choice(["lbvh63", "lbvh30", "hybrid", "sah4"])
        hi = {"lbvh63": 16777216, "lbvh30": 16777216, "hybrid": 5000000, "sah4": 2000000}[preset]
        return dict(kind=kind, scene=rng.choice(["soup", "mesh", "spheres"]), n=_log_int(rng, 20000, hi), preset=preset)
    if kind == "trace":
        return dict(kind=kind, scene=rng.choice(["soup", "mesh", "spheres"]), n=_log_int(rng, 1000, 2000000),
                    preset=rng.choice(["hybrid", "lbvh63", "lbvh30", "sah4"]), rays=rng.choice(["inside", "outside"]),
                    n_rays=_log_int(rng, 500, 4194304), flags=rng.choice([0, 0, 1, 2]))
    if kind == "camera":
        w = _log_int(rng, 300, 1920)
        return dict(kind=kind, scene=rng.choice(["mesh", "spheres"]), n=_log_int(rng, 5000, 2000000),
                    preset=rng.choice(["hybrid", "lbvh63", "sah4"]), width=w, height=max(1, w * rng.randint(50, 100) // 100))
    w = _log_int(rng, 100, 1024)
    h = max(1, w * rng.randint(50, 100) // 100)
    if kind == "render":
        return dict(kind=kind, scene=rng.choice(["cornell", "spheres"]), n=_log_int(rng, 5000, 2000000),
                    preset=rng.choice(["hybrid", "lbvh30", "sah4"]), width=w, height=h, spp=_log_int(rng, 1, 65),
                    max_bounce=rng.randint(2, 8), rr_after=rng.choice([-1, 2]), wavefront=rng.random() < 0.6)
    if kind == "batch":
        w = min(w, 512)
        return dict(kind=kind, n_scenes=rng.randint(2, 64), lo=1000, hi=_log_int(rng, 2000, 300000), width=w, height=min(h, w),
                    spp=rng.randint(1, 8), max_bounce=rng.randint(2, 6), preset=rng.choice(["lbvh30", "hybrid"]))
    w = min(w, 512)
    return dict(kind="diff", n=_log_int(rng, 1000, 200000), preset=rng.choice(["hybrid", "lbvh30"]), width=w, height=min(h, w),
                spp=_log_int(rng, 1, 33), max_bounce=rng.randint(2, 5))


# ---- geometry (positions and normals (V, 6) float32, indices (N, 3) int32, on the GPU) ---------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _soup(n, g):
    """Centroids uniform in the unit cube, vertices at log-uniform distances in [1e-4, 1e-2]."""
    verts = torch.empty(n, 3, 6, device="cuda")
    for a in range(0, n, 1 << 21):
        m = min(1 << 21, n - a)
        c = torch.rand(m, 1, 3, generator=g, device="cuda", dtype=torch.float64)
        ln = torch.exp(torch.rand(m, 3, 1, generator=g, device="cuda", dtype=torch.float64) * math.log(100.0) + math.log(1e-4))
        u = torch.randn(m, 3, 3, generator=g, device="cuda", dtype=torch.float64)
        p = (c + ln * u / u.norm(dim=2, keepdim=True)).float()
        e = p.double()
        nrm = torch.linalg.cross(e[:, 1] - e[:, 0], e[:, 2] - e[:, 0])
        nrm = nrm / nrm.norm(dim=1, keepdim=True).clamp_min(1e-30)
        verts[a:a + m, :, :3] = p
        verts[a:a + m, :, 3:] = nrm.float()[:, None, :]
    return verts.reshape(-1, 6), torch.arange(3 * n, device="cuda", dtype=torch.int32).reshape(n, 3)


@functools.lru_cache(maxsize=None)
def _unit_sphere(level):
    """The icosahedron after `level` midpoint subdivisions: unit vertices, faces, and up to six
    faces around each vertex (padded with the face count)."""
    t = (1.0 + 5.0 ** 0.5) / 2.0
    v = np.array([[-1, t, 0], [1, t, 0], [-1, -t, 0], [1, -t, 0], [0, -1, t], [0, 1, t], [0, -1, -t], [0, 1, -t],
                  [t, 0, -1], [t, 0, 1], [-t, 0, -1], [-t, 0, 1]], np.float64)
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    f = np.array([[0, 11, 5], [0, 5, 1], [0, 1, 7], [0, 7, 10], [0, 10, 11], [1, 5, 9], [5, 11, 4], [11, 10, 2], [10, 7, 6],
                  [7, 1, 8], [3, 9, 4], [3, 4, 2], [3, 2, 6], [3, 6, 8], [3, 8, 9], [4, 9, 5], [2, 4, 11], [6, 2, 10],
                  [8, 6, 7], [9, 8, 1]], np.int64)
    for _ in range(level):
        e = np.sort(f[:, [0, 1, 1, 2, 2, 0]].reshape(-1, 2), axis=1)
        key, inv = np.unique(e[:, 0] * len(v) + e[:, 1], return_inverse=True)
        m = v[key // len(v)] + v[key % len(v)]
        mid = (inv + len(v)).reshape(-1, 3)
        v = np.concatenate([v, m / np.linalg.norm(m, axis=1, keepdims=True)])
        f = np.concatenate([np.stack([f[:, 0], mid[:, 0], mid[:, 2]], 1), np.stack([f[:, 1], mid[:, 1], mid[:, 0]], 1),
                            np.stack([f[:, 2], mid[:, 2], mid[:, 1]], 1), mid], 1).reshape(-1, 3)
    corner = f.reshape(-1)
    order = np.argsort(corner, kind="stable")
    first = np.searchsorted(corner[order], np.arange(len(v)))
    around = np.full((len(v), 6), len(f), np.int64)
    around[corner[order], np.arange(len(corner)) - first[corner[order]]] = order // 3
    return tuple(torch.from_numpy(x).cuda() for x in (v, f[:, [0, 2, 1]].copy(), around))


def _sphere_mesh(n, g, center=(0.0, 0.0, 0.0), radius=1.0):
    """The first n faces of a sphere whose vertices are pushed radially by up to 5 %, with smooth
    normals; wound so that rays from outside hit it."""
    level = 0
    while 20 * 4 ** level < n:
        level += 1
    v, f, around = _unit_sphere(level)
    push = 1.0 + 0.05 * (2.0 * torch.rand(v.shape[0], 1, generator=g, device="cuda", dtype=torch.float64) - 1.0)
    p = v * push * radius + torch.tensor(center, device="cuda", dtype=torch.float64)
    fn = torch.linalg.cross(p[f[:, 2]] - p[f[:, 0]], p[f[:, 1]] - p[f[:, 0]])
    nrm = torch.cat([fn, torch.zeros(1, 3, device="cuda", dtype=torch.float64)])[around].sum(dim=1)
    nrm = nrm / nrm.norm(dim=1, keepdim=True)
    return torch.cat([p, nrm], dim=1).float(), f[:n].int()


def _quad(p, normal):
    e1, e2 = np.subtract(p[1], p[0]), np.subtract(p[2], p[0])
    if np.dot(np.cross(e1, e2), normal) > 0:
        p = [p[0], p[3], p[2], p[1]]
    v = torch.tensor([list(map(float, q)) + list(map(float, normal)) for q in p], device="cuda")
    return v, torch.tensor([[0, 1, 2], [0, 2, 3]], device="cuda", dtype=torch.int32)


def _join(parts):
    vs, ts, ids, off = [], [], [], 0
    for i, (v, t) in enumerate(parts):
        vs.append(v)
        ts.append(t + off)
        ids.append(torch.full((t.shape[0],), i, device="cuda", dtype=torch.int32))
        off += v.shape[0]
    return torch.cat(vs), torch.cat(ts), torch.cat(ids)


def _mat(albedo, emission=(0.0, 0.0, 0.0), kind=0):
    return dict(albedo=tuple(map(float, albedo)), emission=tuple(map(float, emission)), kind=kind)


def _box_parts():
    """A Cornell box with an open front and its quad light."""
    q = [([(-1, -1, -1), (1, -1, -1), (1, -1, 1), (-1, -1, 1)], (0, 1, 0)), ([(-1, 1, -1), (1, 1, -1), (1, 1, 1), (-1, 1, 1)], (0, -1, 0)),
         ([(-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1)], (0, 0, -1)), ([(-1, -1, -1), (-1, -1, 1), (-1, 1, 1), (-1, 1, -1)], (1, 0, 0)),
         ([(1, -1, -1), (1, -1, 1), (1, 1, 1), (1, 1, -1)], (-1, 0, 0)),
         ([(-0.25, 0.998, -0.25), (0.25, 0.998, -0.25), (0.25, 0.998, 0.25), (-0.25, 0.998, 0.25)], (0, -1, 0))]
    mats = [_mat((0.75,) * 3)] * 3 + [_mat((0.65, 0.1, 0.1)), _mat((0.1, 0.6, 0.15)), _mat((0.0,) * 3, (15.0,) * 3)]
    return [_quad(*x) for x in q], mats


def _floor_and_lights(n_lights):
    parts = [_quad([(-1, -0.05, -1), (2, -0.05, -1), (2, -0.05, 2), (-1, -0.05, 2)], (0, 1, 0))]
    mats = [_mat((0.6,) * 3)]
    for k in range(n_lights):
        x, z = (0.5, 0.5) if n_lights == 1 else ((0.15, 0.85)[k % 2], (0.15, 0.85)[k // 2])
        parts.append(_quad([(x - 0.2, 1.6, z - 0.2), (x + 0.2, 1.6, z - 0.2), (x + 0.2, 1.6, z + 0.2), (x - 0.2, 1.6, z + 0.2)], (0, -1, 0)))
        mats.append(_mat((0.0,) * 3, (20.0, 18.0 + 2 * k, 16.0)))
    return parts, mats


BOX_VIEW = ((0.0, 0.0, -3.4), (0.0, 0.0, 0.0), 40.0)
ROOM_VIEW = ((0.5, 0.9, -1.6), (0.5, 0.35, 0.5), 45.0)


def _scene(kind, n, seed):
    """(verts, tris, material per input triangle, materials, camera) of about n triangles."""
    g = _gen(seed)
    rng = np.random.default_rng(seed)
    if kind == "soup":
        v, t = _soup(n, g)
        return v, t, torch.zeros(n, device="cuda", dtype=torch.int32), [_mat(rng.uniform(0.2, 0.8, 3))], ROOM_VIEW
    if kind == "mesh":
        v, t = _sphere_mesh(n, g, (0.5, 0.5, 0.5), 0.45)
        return v, t, torch.zeros(n, device="cuda", dtype=torch.int32), [_mat(rng.uniform(0.2, 0.8, 3))], ROOM_VIEW
    if kind == "cornell":
        parts, mats = _box_parts()
        parts.append(_sphere_mesh(n, g, (0.15, -0.45, 0.25), 0.5))
        parts += [_sphere_mesh(960, g, c, 0.3) for c in ((-0.55, -0.7, -0.35), (0.6, -0.7, -0.5))]
        mats = mats + [_mat((a,) * 3) for a in rng.uniform(0.2, 0.8, 3)]
        v, t, m = _join(parts)
        return v, t, m, mats, BOX_VIEW
    # "spheres": many spheres of uneven sizes, four fifths diffuse and one fifth mirrors
    count = max(8, min(400, n // 1000))
    each = max(1, n // count)
    parts, mats = [], []
    for k in range(count):
        r = math.exp(rng.uniform(math.log(0.01), math.log(0.2)))
        parts.append(_sphere_mesh(each, g, tuple(rng.uniform(0.0, 1.0, 3)), r))
        mats.append(_mat((0.9,) * 3, kind=1) if rng.random() < 0.2 else _mat(rng.uniform(0.2, 0.8, 3)))
    fp, fm = _floor_and_lights(4)
    v, t, m = _join(parts + fp)
    return v, t, m, mats + fm, ROOM_VIEW


def _rays(kind, n, lo, hi, g):
    """Origins uniform in the box (or on a sphere around it), directions uniform (or into the box)."""
    lo, hi = lo.double(), hi.double()
    o = lo + (hi - lo) * torch.rand(n, 3, generator=g, device="cuda", dtype=torch.float64)
    d = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    d = d / d.norm(dim=1, keepdim=True)
    if kind == "outside":
        start = (lo + hi) / 2 + d * (hi - lo).norm()
        d = o - start
        o, d = start, d / d.norm(dim=1, keepdim=True)
    r = torch.zeros(n, 8, device="cuda")
    r[:, 0:3] = o
    r[:, 4:7] = d
    r[:, 7] = INF
    return r


def _camera_rays(width, height, view):
    pos, target, fov = (torch.tensor(x, device="cuda", dtype=torch.float64) for x in view)
    fwd = target - pos
    fwd = fwd / fwd.norm()
    right = torch.linalg.cross(fwd, torch.tensor([0.0, 1.0, 0.0], device="cuda", dtype=torch.float64))
    right = right / right.norm()
    up = torch.linalg.cross(right, fwd)
    th = torch.tan(torch.deg2rad(fov) * 0.5)
    x = ((torch.arange(width, device="cuda", dtype=torch.float64) + 0.5) / width * 2 - 1) * (width / height) * th
    y = ((torch.arange(height, device="cuda", dtype=torch.float64) + 0.5) / height * 2 - 1) * th
    d = (fwd + x[None, :, None] * right + y[:, None, None] * up).reshape(-1, 3)
    r = torch.zeros(width * height, 8, device="cuda")
    r[:, 0:3] = pos
    r[:, 3] = 1e-3
    r[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    r[:, 7] = INF
    return r


# ---- preparing and running ----------------------------------------------------------------------

def _materials(mats):
    return torch.from_numpy(rtb200.materials_array(mats)).cuda()


def _baked(per_input_triangle, bvh):
    """A per-triangle table in the order of the baked triangles."""
    return per_input_triangle[torch.from_numpy(bvh.prim_ids().astype(np.int64)).cuda()].contiguous()


def _batch_counts(case):
    k = np.linspace(math.log(case["lo"]), math.log(case["hi"]), case["n_scenes"])
    return np.random.default_rng(3).permutation(np.exp(k).astype(np.int64))


def _batch_parts(case, seed):
    """Scenes that are a sphere or a soup by turns, each over a floor and under one light."""
    g = _gen(seed)
    fp, fm = _floor_and_lights(1)
    rng = np.random.default_rng(seed)
    parts, mats, mot = [], [], []
    for s, n in enumerate(_batch_counts(case)):
        body = _sphere_mesh(int(n), g, (0.5, 0.45, 0.5), 0.4) if s % 2 == 0 else _soup(int(n), g)
        v, t, m = _join([body] + fp)
        parts.append((v, t))
        mot.append(m + len(mats))
        mats += [_mat(rng.uniform(0.2, 0.8, 3))] + fm
    return parts, mats, torch.cat(mot)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        parts, mats, mot = _batch_parts(case, seed)
        st = dict(case=case, verts=torch.cat([v for v, _ in parts]), tris=torch.cat([t for _, t in parts]),
                  vo=np.cumsum([0] + [v.shape[0] for v, _ in parts]).astype(np.uint32),
                  to=np.cumsum([0] + [t.shape[0] for _, t in parts]).astype(np.uint32), cfg=rtb200.make_cfg(case["preset"]))
        st["bvh"] = rtb200.Bvh.build_batch(st["verts"], st["tris"], st["vo"], st["to"], st["cfg"])
        st["mats"], st["mot"] = _materials(mats), _baked(mot, st["bvh"])
        st["rcfgs"] = [rtb200.render_cfg(case["width"], case["height"], case["spp"], max_bounce=case["max_bounce"], rr_after=-1, env_kind=1,
                                         env_color=(0.02, 0.02, 0.03), seed=seed * 100 + s, lookat=ROOM_VIEW) for s in range(case["n_scenes"])]
        return st
    if kind == "diff":
        verts, tris, mot, mats, view = _scene("cornell", case["n"], seed)
        bvh = rtb200.Bvh.build(verts, tris, case["preset"])
        g = _gen(seed + 1)
        return dict(case=case, bvh=bvh, mats=_materials(mats), mot=_baked(mot, bvh),
                    albedo=0.2 + 0.6 * torch.rand(tris.shape[0], 3, generator=g, device="cuda"),
                    target=torch.rand(case["height"], case["width"], 3, generator=g, device="cuda"),
                    rcfg=rtb200.render_cfg(case["width"], case["height"], case["spp"], max_bounce=case["max_bounce"], rr_after=-1, env_kind=1,
                                           seed=seed, lookat=view))
    verts, tris, mot, mats, view = _scene(case["scene"], case["n"], seed)
    st = dict(case=case, cfg=rtb200.make_cfg(case["preset"]))
    if kind == "bake_host":
        st["verts"], st["tris"] = verts.cpu(), tris.cpu()
        if case["pinned"]:
            st["verts"], st["tris"] = st["verts"].pin_memory(), st["tris"].pin_memory()
        st["nv"], st["nt"] = st["verts"].numpy(), st["tris"].numpy().view(np.uint32)
        st["bvh"] = rtb200.Bvh.build(st["nv"], st["nt"], st["cfg"])
        # the caller's buffers for the baked arrays, with room for the references of spatial splits
        out = [torch.zeros(4 * case["n"], 48, dtype=torch.uint8), torch.zeros(2 * case["n"], 3, dtype=torch.int32),
               torch.zeros(verts.shape[0], 6)]
        st["keep"] = [x.pin_memory() for x in out] if case["pinned"] else out
        st["nodes"] = st["keep"][0].numpy().view(rtb200.NODE_DTYPE).reshape(-1)
        return st
    st["bvh"] = rtb200.Bvh.build(verts, tris, st["cfg"])
    if kind == "bake":
        st["verts"], st["tris"] = verts, tris
        st["prim"] = torch.zeros(2 * case["n"] + 64, device="cuda", dtype=torch.int32)
    elif kind == "trace":
        lo, hi = verts[:, :3].min(dim=0).values, verts[:, :3].max(dim=0).values
        st["rays"] = _rays(case["rays"], case["n_rays"], lo, hi, _gen(seed + 2))
    elif kind == "camera":
        st["rays"] = _camera_rays(case["width"], case["height"], view)
        st["rays"][:, 0:3] += 0.01 * torch.randn(3, generator=_gen(seed + 2), device="cuda")
        hits = st["bvh"].trace(st["rays"])
        hit = hits.view(torch.int32)[:, 7:8] & 1
        at = st["rays"][:, 0:3] + st["rays"][:, 4:7] * hits[:, 0:1]
        to = torch.tensor([0.5, 1.55, 0.5], device="cuda") - at
        far = to.norm(dim=1, keepdim=True)
        # shadow rays towards a point under the lights; pixels that see nothing ask about their own ray
        shadow = torch.cat([at, torch.full_like(far, 1e-3), to / far, far * 0.999], dim=1)
        st["shadow"] = torch.where(hit != 0, shadow, st["rays"]).contiguous()
    elif kind == "render":
        st["mats"], st["mot"] = _materials(mats), _baked(mot, st["bvh"])
        st["rcfg"] = rtb200.render_cfg(case["width"], case["height"], case["spp"], max_bounce=case["max_bounce"], rr_after=case["rr_after"],
                                       env_kind=1, env_color=(0.02, 0.02, 0.03), seed=seed, lookat=view)
    return st


def _ok(code):
    if code != 0:
        raise rtb200.RtError(code, rtb200.last_error())


def _hits(h):
    """The records of a trace as their fields: distance and barycentrics, triangle, normal, flags."""
    w = h.view(torch.int32)
    return {"tuv": h[:, 0:3], "tri": w[:, 3], "normal": h[:, 4:7], "flags": w[:, 7]}


def run(state):
    case, bvh = state["case"], state["bvh"]
    kind = case["kind"]
    if kind == "bake_host":
        bvh.rebuild(state["nv"], state["nt"], state["cfg"])
        lib, nodes, (_, tris, verts) = rtb200.lib(), state["nodes"], state["keep"]
        if case["pinned"]:
            _ok(lib.rt_bvh_download_async(bvh.h, nodes.ctypes.data, tris.data_ptr(), verts.data_ptr(), None))
            _ok(lib.rt_device_sync(None))
        else:
            _ok(lib.rt_bvh_download(bvh.h, nodes.ctypes.data, tris.data_ptr(), verts.data_ptr()))
        nn, nt, _ = bvh.counts()
        return {"lo": nodes["bmin"], "hi": nodes["bmax"], "is_leaf": nodes["is_leaf"], "a": nodes["a"].view(np.int32),
                "b": nodes["b"].view(np.int32), "tris": tris, "verts": verts, "n_nodes": nn, "n_tris": nt}
    if kind == "bake":
        bvh.rebuild(state["verts"], state["tris"], state["cfg"])
        nn, nt, _ = bvh.counts()
        # the order of the baked triangles, for the caller's per-triangle tables
        _ok(rtb200.lib().rt_bvh_prim_ids(bvh.h, state["prim"].data_ptr(), 1))
        return {"prim": state["prim"], "nodes": nn, "tris": nt, "stats": bvh.stats()}
    if kind == "trace":
        return _hits(bvh.trace(state["rays"], case["flags"]))
    if kind == "camera":
        return {"seen": _hits(bvh.trace(state["rays"])), "shadow": _hits(bvh.trace(state["shadow"], rtb200.TRACE_ANY_HIT))}
    if kind == "render":
        mode = rtb200.RENDER_WAVEFRONT if case["wavefront"] else rtb200.RENDER_PLAIN
        return bvh.render(state["rcfg"], state["mats"], state["mot"], mode)[0]
    if kind == "batch":
        bvh.rebuild_batch(state["verts"], state["tris"], state["vo"], state["to"], state["cfg"])
        return bvh.render_batch(state["rcfgs"], state["mats"], state["mot"])[0]
    # a step of inverse rendering: image, the L2 loss's gradient, and the adjoint
    rgb = bvh.render(state["rcfg"], state["mats"], state["mot"], tri_albedo=state["albedo"])[0]
    g_albedo, g_emission = bvh.adjoint(state["rcfg"], 2.0 * (rgb - state["target"]), state["mats"], state["mot"], tri_albedo=state["albedo"])
    return {"rgb": rgb, "g_albedo": g_albedo, "g_emission": g_emission}


# ---- what a pass cannot do without ---------------------------------------------------------------

def _vertices(scene, n):
    return 3 * n if scene == "soup" else n // 2 + 2


def _tree_bytes(n, preset):
    """A two-child node per inner node and a triangle's positions, each read once."""
    return n / LEAF[preset] * 48 + 36 * n


def _trace_flops(n, preset):
    """One ray: two box tests per level and twice (the near and one far subtree) a leaf's triangles."""
    return max(1.0, math.log2(n / LEAF[preset] + 1)) * 2 * 24 + 2 * LEAF[preset] * 45


def work(case):
    kind, preset = case["kind"], case["preset"]
    if kind in ("bake", "bake_host"):
        n = case["n"]
        v = _vertices(case["scene"], n)
        # vertices and triangles in; nodes, triangles, ids and vertices out; about 60 operations per
        # triangle and level of quantisation or binning
        return {"bytes": 48.0 * v + 28.0 * n + 96.0 * n / LEAF[preset],
                "flops": 60.0 * n * (1 if preset.startswith("lbvh") else max(1.0, math.log2(n / LEAF[preset] + 1)))}
    if kind in ("trace", "camera"):
        rays = case["n_rays"] if kind == "trace" else 2 * case["width"] * case["height"]
        return {"bytes": 64.0 * rays + _tree_bytes(case["n"], preset), "flops": rays * _trace_flops(case["n"], preset)}
    px = case["width"] * case["height"]
    if kind == "batch":
        n = int(_batch_counts(case).sum())
        rays = px * case["n_scenes"] * case["spp"] * 1.2
        return {"bytes": 12.0 * px * case["n_scenes"] + 172.0 * n, "flops": 60.0 * n + rays * (_trace_flops(n / case["n_scenes"], preset) + 150)}
    # paths of a closed box run to the last bounce, those over the open floor leave after two
    deep = case["max_bounce"] + 1 if kind == "diff" or case["scene"] == "cornell" else min(2, case["max_bounce"] + 1)
    passes = 2 if kind == "diff" else 1  # the image, and its paths once more for the gradients
    rays = px * case["spp"] * deep * passes
    return {"bytes": 12.0 * px * (3 if kind == "diff" else 1) + _tree_bytes(case["n"], preset) + (24.0 * case["n"] if kind == "diff" else 0.0),
            "flops": rays * (_trace_flops(case["n"], preset) + 150)}


# ---- the same results in 64 bits -------------------------------------------------------------------

def _exact_hits(verts, tris, rays):
    """Closest front-facing hits by testing every triangle, in double precision."""
    v = verts.double()
    p0, p1, p2 = (v[tris[:, k].long(), :3] for k in range(3))
    e1, e2 = p1 - p0, p2 - p0
    tuv = torch.zeros(rays.shape[0], 3, device="cuda", dtype=torch.float64)
    normal = torch.zeros_like(tuv)
    step = max(1, (1 << 24) // tris.shape[0])
    for k in range(0, rays.shape[0], step):
        r = rays[k:k + step].double()
        o, d = r[:, None, 0:3], r[:, None, 4:7]
        h = torch.linalg.cross(d.expand(-1, e2.shape[0], -1), e2.expand(d.shape[0], -1, -1))
        a = (e1 * h).sum(-1)
        s = o - p0
        u = (s * h).sum(-1) / a
        q = torch.linalg.cross(s, e1.expand(s.shape[0], -1, -1))
        w = (d * q).sum(-1) / a
        t = (e2 * q).sum(-1) / a
        ok = (a < 0) & (u >= 0) & (u <= 1) & (w >= 0) & (u + w <= 1) & (t >= r[:, None, 3]) & (t <= r[:, None, 7])
        best, at = torch.where(ok, t, INF).min(dim=1)
        got = torch.isfinite(best)
        row = torch.arange(len(at), device="cuda")
        u, w = u[row, at], w[row, at]
        n = v[tris[at, 0].long(), 3:] * (1 - u - w)[:, None] + v[tris[at, 1].long(), 3:] * u[:, None] + v[tris[at, 2].long(), 3:] * w[:, None]
        tuv[k:k + step] = torch.where(got[:, None], torch.stack([best, u, w], 1), 0.0)
        normal[k:k + step] = torch.where(got[:, None], n / n.norm(dim=1, keepdim=True), 0.0)
    return tuv, normal


def exact(case, seed):
    """Baked vertices (renormalised normals) and closest hits of moderate size. Boxes and indices are
    copies and choices, which have no other value in 64 bits; an any-hit ray's answer depends on
    the order of the tree; a path tracer's image is one random outcome, whose paths a tracer in
    64 bits would leave at the first rounding difference."""
    if case["kind"] == "bake_host":
        v = _scene(case["scene"], case["n"], seed)[0].double()
        ln = v[:, 3:].norm(dim=1, keepdim=True)
        v[:, 3:] = torch.where(ln > 1e-6, v[:, 3:] / ln.clamp_min(1e-30), torch.tensor([0.0, 1.0, 0.0], device="cuda", dtype=torch.float64))
        return {"lo": None, "hi": None, "is_leaf": None, "a": None, "b": None, "tris": None, "verts": v, "n_nodes": None, "n_tris": None}
    if case["kind"] == "trace" and case["flags"] == 0 and case["n_rays"] * case["n"] <= 1e10:
        verts, tris, _, _, _ = _scene(case["scene"], case["n"], seed)
        lo, hi = verts[:, :3].min(dim=0).values, verts[:, :3].max(dim=0).values
        tuv, normal = _exact_hits(verts, tris, _rays(case["rays"], case["n_rays"], lo, hi, _gen(seed + 2)))
        return {"tuv": tuv, "tri": None, "normal": normal, "flags": None}
    return None
