"""V-BM3D predictive search: match lists against the oracle, index for index, over both kernels (the
register-blocked one and the general one) and where they meet: window clipping, one and two seeds,
the widest window of a warp, group sizes around a warp's 32 lanes, and tied keys."""
import numpy as np
import pytest

from bm3d_b200 import core, source, synth

pytestmark = pytest.mark.gpu


def clip_of(kind, frames, h, w):
    if kind == "noisy":
        nz, _ = synth.motion_frames(3, frames, h, w, 12.0, planes=1)
        return np.ascontiguousarray(nz, np.float32)
    # few levels: equal keys in most searches
    rng = np.random.default_rng(7)
    return (np.round(rng.random((frames, 1, h, w)) * 3) / 255.0).astype(np.float32)


@pytest.mark.parametrize("kind", ["noisy", "ties"])
@pytest.mark.parametrize("h,w,radius,G,R,ps_num,ps_range,ps_step", [
    (8, 8, 1, 8, 7, 2, 4, 1),          # a single block position
    (23, 41, 2, 8, 7, 2, 5, 1),        # windows clipped on every side, ragged quads
    (37, 29, 1, 16, 5, 1, 6, 1),       # one seed
    (48, 64, 3, 8, 12, 2, 6, 1),       # profile np's search
    (40, 56, 1, 32, 9, 2, 8, 1),       # a list of a warp's width
    (52, 44, 1, 33, 7, 2, 4, 1),       # one longer: general kernel
    (52, 44, 1, 8, 7, 2, 12, 1),       # the widest staged window
    (52, 44, 1, 8, 7, 2, 13, 1),       # one wider: general kernel
    (40, 48, 1, 2, 7, 2, 1, 1),        # smallest group and window
    (40, 48, 1, 8, 7, 3, 4, 1),        # three seeds: general kernel
    (40, 48, 1, 8, 7, 2, 4, 2),        # step 2: general kernel
])
def test_predictive_lists(orc, kind, h, w, radius, G, R, ps_num, ps_range, ps_step):
    frames = min(radius + 2, 4)
    clip = clip_of(kind, frames, h, w)
    args = dict(block_step=5, group_size=G, bm_range=R, radius=radius, ps_num=ps_num, ps_range=ps_range, ps_step=ps_step,
                th_mse=3000.0)
    node = core.bm3d.VBasic(source(clip, "GRAY"), matrix=6, **args)
    node.compute(0, frames)
    p = orc.default_params(0, True, "fast", 10.0, matrix=6, **args)
    for n in range(frames):
        cnt, z, y, x, keys = node.matches(n, G)
        ocnt, oz, oy, ox, ok = orc.vbm3d_matches(p, clip[:, 0], n, threads=4)
        assert np.array_equal(cnt, ocnt)
        m = np.arange(G)[None, :] < cnt[:, None]
        for a, b in ((z, oz), (y, oy), (x, ox), (keys.view(np.int32), ok.view(np.int32))):
            assert np.array_equal(a[m], b[m])
