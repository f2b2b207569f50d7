"""Block matching and plain outputs of the precision values that share the plain path, against the oracle: "fp32", "tf32"
and "tf32_match" give the oracle's match lists (positions, order, keys bit for bit), and "tf32_match" its pictures.

Tolerance of the pictures: the transforms are the oracle's, the order of a pixel's sums differs: at most 2^12 terms, rounding
errors independent, within 2^6 * 2^-24 = 4e-6; the bound used is 2e-5."""
import numpy as np
import pytest

from bm3d_b200 import core, source, synth

pytestmark = pytest.mark.gpu

FORMS = ["fp32", "tf32", "tf32_match"]


def check_lists(orc, node, k, p, img):
    cnt, _, y, x, keys = node.matches(k, p.G)
    ocnt, oy, ox, ok = orc.bm3d_matches(p, img, threads=8)
    assert np.array_equal(cnt, ocnt)
    m = np.arange(p.G)[None, :] < cnt[:, None]
    assert np.array_equal(y[m], oy[m]) and np.array_equal(x[m], ox[m])
    assert np.array_equal(keys[m].view(np.int32), ok[m].view(np.int32))


def piecewise_constant(h, w):
    """Many zero and equal distances: lists that the estimates cannot settle."""
    rng = np.random.default_rng(62)
    img = np.zeros((1, 1, h, w), np.float32)
    for _ in range(12):
        y, x = rng.integers(0, h - 16), rng.integers(0, w - 18)
        img[0, 0, y:y + rng.integers(8, 40), x:x + rng.integers(8, 40)] = rng.integers(0, 8) / 8.0
    return img


@pytest.mark.parametrize("precision", FORMS)
@pytest.mark.parametrize("profile,sigma", [("np", 10.0), ("lc", 25.0), ("high", 15.0)])
@pytest.mark.parametrize("h,w", [(160, 224), (40, 56)])
def test_lists(orc, precision, profile, sigma, h, w):
    nz, clean = synth.gray_frames(61, 2, h, w, sigma)
    ref = (clean + np.random.default_rng(8).normal(0, 0.15 * sigma / 255.0, clean.shape)).astype(np.float32)
    kw = dict(profile=profile, sigma=sigma, matrix=6, precision=precision)
    basic = core.bm3d.Basic(source(nz, "GRAY"), **kw)
    final = core.bm3d.Final(source(nz, "GRAY"), source(ref, "GRAY"), **kw)
    for wiener, node, img in ((0, basic, nz), (1, final, ref)):
        node.compute(0, 2)
        p = orc.default_params(wiener, False, profile, sigma, matrix=6)
        for k in range(2):
            check_lists(orc, node, k, p, img[k, 0])


@pytest.mark.parametrize("precision", FORMS)
@pytest.mark.parametrize("wiener", [0, 1])
def test_lists_of_ties(orc, precision, wiener):
    img = piecewise_constant(96, 128)
    kw = dict(profile="np", matrix=6, precision=precision)
    src = source(img, "GRAY")
    node = core.bm3d.Final(src, src, **kw) if wiener else core.bm3d.Basic(src, **kw)
    node.compute(0, 1)
    check_lists(orc, node, 0, orc.default_params(wiener, False, "np", 10.0, matrix=6), img[0, 0])
    assert node.bm_tc_counts()[0] > 0                   # lists settled by exact distances


def test_pictures_of_tf32_match(orc):
    nz, clean = synth.gray_frames(57, 2, 96, 120, 10.0)
    ref = (clean + np.random.default_rng(8).normal(0, 0.006, clean.shape)).astype(np.float32)
    kw = dict(profile="np", matrix=6, precision="tf32_match")
    basic = core.bm3d.Basic(source(nz, "GRAY"), **kw).numpy()
    final = core.bm3d.Final(source(nz, "GRAY"), source(ref, "GRAY"), **kw).numpy()
    for wiener, got in ((0, basic), (1, final)):
        exp = orc.bm3d(orc.default_params(wiener, False, "np", 10.0, matrix=6), nz, ref if wiener else None, threads=8)
        assert np.abs(got - exp).max() <= 2e-5
