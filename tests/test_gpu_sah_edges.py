"""SAH builds at the node sizes where the builder changes kernels (64, 512, 2,048 references, chunks of
1,024) and on triangles that fan around shared vertices, whose spatial splits straddle on several axes.
Bar: the oracle's tree."""
import numpy as np
import pytest

import rtb200
from rtb200 import scenes
from oracle import make_cfg as orc_make_cfg
from test_gpu_build import assert_same_tree, orc_cfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [63, 64, 65, 511, 513, 1023, 1025, 2047, 2048, 2049, 3073, 4097, 9000])
@pytest.mark.parametrize("kind", ["soup", "mesh"])
def test_sizes(orc, n, kind):
    if kind == "soup":
        v, t = scenes.soup(n, seed=n, lo=1e-3, hi=3e-1)
    else:
        v, t = scenes.icosphere(5, seed=n, max_tris=n)
    b = rtb200.Bvh.build(v, t, "sah4")
    assert_same_tree(b.download(), orc.build(v, t, orc_cfg("sah4")), f"{kind}/{n}")


def fans(count, blades, seed):
    """Fans of long thin triangles around shared vertices, tilted at random."""
    rng = np.random.default_rng(seed)
    vs, ts = [], []
    for k in range(count):
        c = rng.uniform(0, 1, 3)
        q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        a = np.linspace(0, 2 * np.pi, blades, endpoint=False)
        rim = c + 0.3 * (np.cos(a)[:, None] * q[0] + np.sin(a)[:, None] * q[1] + 0.2 * rng.normal(size=(blades, 1)) * q[2])
        base = sum(x.shape[0] for x in vs)
        vs.append(np.concatenate([c[None], rim]))
        i = np.arange(blades)
        ts.append(np.stack([np.zeros(blades, int), 1 + i, 1 + (i + 1) % blades], 1) + base)
    p = np.concatenate(vs)
    v = np.zeros((p.shape[0], 6), np.float32)
    v[:, :3] = p
    v[:, 4] = 1.0
    return v, np.concatenate(ts).astype(np.uint32)


@pytest.mark.parametrize("preset", ["hybrid", "sah4", "sah16"])
@pytest.mark.parametrize("count,blades", [(1, 17), (1, 60), (12, 24), (60, 33)])
def test_fans(orc, preset, count, blades):
    v, t = fans(count, blades, 3)
    b = rtb200.Bvh.build(v, t, preset)
    ref = orc.build(v, t, orc_cfg(preset))
    assert_same_tree(b.download(), ref, f"{preset}/{count}x{blades}")
    assert b.stats()["spatial_taken"] == int(ref.stats[0])


@pytest.mark.parametrize("mult", [1.0, 1.01, 1.1, 1.5])
@pytest.mark.parametrize("count,blades", [(12, 24), (300, 33), (900, 40)])
def test_budgets(orc, count, blades, mult):
    """Reference budgets that no, some, or all spatial splits of a level fit, on levels within one block's reach
    (4,096 nodes) and beyond it."""
    v, t = fans(count, blades, 5)
    b = rtb200.Bvh.build(v, t, rtb200.make_cfg("sah4", spatial_mult=mult))
    ref = orc.build(v, t, orc_make_cfg(**{**rtb200.PRESETS["sah4"], "spatial_mult": mult}))
    assert_same_tree(b.download(), ref, f"{count}x{blades}/{mult}")
    st = b.stats()
    assert st["spatial_taken"] == int(ref.stats[0]) and st["spatial_refused"] == int(ref.stats[1])


@pytest.mark.parametrize("n", [65, 2000, 44000, 52000, 56000, 70000])
def test_root_counts(orc, n):
    """Hybrid bakes of one to some 1,500 SAH subtrees (one block orders up to 1,024)."""
    v, t = scenes.soup(n, seed=n, lo=1e-3, hi=1e-1)
    b = rtb200.Bvh.build(v, t, "hybrid")
    assert_same_tree(b.download(), orc.build(v, t, orc_cfg("hybrid")), f"hybrid/{n}")
