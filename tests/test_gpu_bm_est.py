"""Full search with shared estimates and an exact short list: match lists index for index (positions,
order, keys bit for bit) against the oracle, over the block steps and ranges it takes, ragged rows of
reference blocks, frames smaller than the window, short, empty and tied lists, flat areas, and ranges on
either side of what fits."""
import numpy as np
import pytest

from bm3d_b200 import core, source, synth

pytestmark = pytest.mark.gpu


def check(orc, img, **over):
    node = core.bm3d.Basic(source(np.ascontiguousarray(img, np.float32)[None, None], "GRAY"), profile="np", matrix=6, **over)
    node.compute(0, 1)
    p = orc.default_params(0, False, "np", 10.0, matrix=6, **over)
    cnt, _, y, x, keys = node.matches(0, p.G)
    ocnt, oy, ox, ok = orc.bm3d_matches(p, img.astype(np.float32), threads=8)
    assert np.array_equal(cnt, ocnt)
    m = np.arange(p.G)[None, :] < cnt[:, None]
    assert np.array_equal(y[m], oy[m]) and np.array_equal(x[m], ox[m])
    assert np.array_equal(keys[m].view(np.int32), ok[m].view(np.int32))
    return node, cnt


def noisy(h, w, seed=5):
    return synth.gray_frames(seed, 1, h, w, 10.0)[0][0, 0]


@pytest.mark.parametrize("step", range(1, 9))
@pytest.mark.parametrize("R,G", [(16, 16), (9, 32), (3, 8)])
def test_steps_and_ranges(orc, step, R, G):
    check(orc, noisy(45, 71), block_step=step, bm_range=R, group_size=G)


@pytest.mark.parametrize("h,w", [(8, 8), (8, 60), (60, 9), (33, 32), (40, 97), (41, 98), (42, 99), (43, 100)])
def test_frame_sizes(orc, h, w):
    check(orc, noisy(h, w), block_step=3, group_size=32)


@pytest.mark.parametrize("th", [0.5, 20.0, 150.0, 1e6])
def test_thresholds(orc, th):
    """Empty, short and complete lists, and every candidate below the threshold."""
    check(orc, noisy(48, 64), th_mse=th)


@pytest.mark.parametrize("R", [40, 60])
def test_large_ranges(orc, R):
    """The largest windows of this search, and one beyond it (the exact search takes it)."""
    check(orc, noisy(60, 90), bm_range=R, block_step=8)


def test_quantised_pictures(orc):
    """Integer sample values: equal keys in many lists and at many cuts."""
    img = np.round(noisy(64, 96) * 255.0) / 255.0
    check(orc, img, group_size=32)
    img = np.round(noisy(64, 96) * 31.0) / 31.0
    node, _ = check(orc, img)
    assert node.bm_tc_counts()[0] > 0


def test_flat_areas(orc):
    """Letterbox bars: all distances inside them are zero, which is no match."""
    img = noisy(96, 80)
    img[:32] = 0.0
    img[-24:] = 0.0
    _, cnt = check(orc, img, block_step=4)
    assert (cnt[:19 * 3] == 1).all()        # rows of blocks (19 each) whose windows lie in the top bar


@pytest.mark.parametrize("scale", [1e-15, 1e-4, 1e6])
def test_scales(orc, scale):
    check(orc, noisy(48, 56) * scale, th_mse=2000.0 * scale * scale)


def test_nan_pixels(orc):
    img = noisy(48, 64)
    img[20, 30] = np.nan
    check(orc, img)
