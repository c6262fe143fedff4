"""Large bakes sort the top four digits of their codes and then runs of equal ones; crowded inputs
and runs above n / 512 that a sample of the keys misses fall back to all digits. The bar is the
oracle's stable Morton order for each."""
import numpy as np
import pytest

import rtb200
from oracle import make_cfg as orc_make_cfg
from rtb200 import scenes

pytestmark = pytest.mark.gpu

N = (1 << 21) + 1000
SAMPLES = 8192


def crowd(v, which, seed):
    """The triangles `which`, shrunk into one 4,096th of the scene's box."""
    rng = np.random.default_rng(seed)
    v = v.copy().reshape(-1, 3, 6)
    lo, hi = v[:, :, :3].min((0, 1)), v[:, :, :3].max((0, 1))
    c = lo + (hi - lo) * (np.array([800.5, 700.5, 300.5], np.float32) / 2048)
    p = c + (hi - lo) * rng.uniform(-1 / 8192, 1 / 8192, (len(which), 1, 3))
    v[which, :, :3] = p + (hi - lo) * 1e-6 * rng.uniform(-1, 1, (len(which), 3, 3))
    return v.reshape(-1, 6)


@pytest.mark.parametrize("bits", [21, 17])
@pytest.mark.parametrize("case", ["soup", "long_run", "missed_run", "crowded"])
def test_order(orc, case, bits):
    v, t = scenes.soup(N, seed=85)
    rng = np.random.default_rng(86)
    sampled = np.arange(SAMPLES, dtype=np.int64) * N // SAMPLES
    unsampled = rng.permutation(np.setdiff1d(np.arange(N), sampled))
    if case == "long_run":
        v = crowd(v, unsampled[: N // 512 - 40], 87)
    elif case == "missed_run":
        v = crowd(v, unsampled[: N // 512 + 40], 88)
    elif case == "crowded":
        v = crowd(v, rng.permutation(N)[:20000], 89)
    kw = dict(rtb200.PRESETS["lbvh63"], morton_bits=bits)
    codes, perm, _ = orc.morton(v, t, orc_make_cfg(**kw))
    codes = np.sort(np.asarray(codes, np.uint64))
    top = codes >> np.uint64(8 * ((3 * bits + 7) // 8 - 4))
    longest = int(np.unique(top, return_counts=True)[1].max())
    assert (longest > N // 512) == (case in ("missed_run", "crowded"))
    pid = rtb200.Bvh.build(v, t, rtb200.make_cfg(**kw)).prim_ids()
    # runs of more identical codes than a leaf holds are reordered by their SAH subtree
    loose = np.unique(codes, return_inverse=True, return_counts=True)
    loose = loose[2][loose[1]] > kw["max_leaf"]
    assert np.mean(loose) < 0.01
    assert np.array_equal(pid[~loose], perm[~loose])
