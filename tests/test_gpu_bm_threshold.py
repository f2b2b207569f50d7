"""Match lists under huge thresholds ("every candidate matches"): thresholds that stay finite in fp32, that
overflow there, and infinite ones, over search windows small enough that a group takes all of their
candidates, and pictures whose distances overflow.  Index for index against the oracle, keys bit for bit."""
import numpy as np
import pytest

from bm3d_b200 import core, source, synth

pytestmark = pytest.mark.gpu

THRESHOLDS = [1e37, 3e40, 3e41, 1e300, float("inf")]


def same_lists(got, exp, G):
    cnt = got[0]
    assert np.array_equal(cnt, exp[0])
    m = np.arange(G)[None, :] < cnt[:, None]
    for a, b in zip(got[1:-1], exp[1:-1]):
        assert np.array_equal(a[m], b[m])
    assert np.array_equal(got[-1][m].view(np.int32), exp[-1][m].view(np.int32))


@pytest.mark.parametrize("th", THRESHOLDS)
@pytest.mark.parametrize("R,G,step", [(1, 16, 4), (2, 16, 3), (3, 32, 8), (4, 8, 4), (16, 16, 4)])
@pytest.mark.parametrize("scale", [1.0, 1e20])
def test_full_search(orc, th, R, G, step, scale):
    img = (synth.gray_frames(5, 1, 37, 46, 10.0)[0][0, 0] * scale).astype(np.float32)
    over = dict(bm_range=R, group_size=G, block_step=step, th_mse=th)
    node = core.bm3d.Basic(source(img[None, None], "GRAY"), profile="np", matrix=6, **over)
    node.compute(0, 1)
    p = orc.default_params(0, False, "np", 10.0, matrix=6, **over)
    cnt, _, y, x, keys = node.matches(0, G)
    same_lists((cnt, y, x, keys), orc.bm3d_matches(p, img, threads=8), G)


@pytest.mark.parametrize("th", THRESHOLDS)
@pytest.mark.parametrize("scale", [1.0, 1e20])
def test_predictive_search(orc, th, scale):
    clip = (synth.motion_frames(3, 3, 29, 38, 12.0, planes=1)[0] * scale).astype(np.float32)
    args = dict(block_step=5, group_size=32, bm_range=2, radius=1, ps_num=2, ps_range=2, ps_step=1, th_mse=th)
    node = core.bm3d.VBasic(source(clip, "GRAY"), matrix=6, **args)
    node.compute(0, 3)
    p = orc.default_params(0, True, "fast", 10.0, matrix=6, **args)
    for n in range(3):
        same_lists(node.matches(n, 32), orc.vbm3d_matches(p, clip[:, 0], n, threads=4), 32)
