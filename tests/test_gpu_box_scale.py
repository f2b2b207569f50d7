"""Plain Basic filter on clips of any magnitude, against the oracle: the filter is scale-free (pixels, sigma and the
square root of th_mse scaled together), so its relative error is too.

Tolerance: both sides run the same transforms; they differ in the order of the sums of a pixel's terms.  A pixel takes
at most 2^12 terms: rounding errors being independent, within 2^6 * 2^-24 = 4e-6 of the value range; the bound used is
2e-5 of the oracle's largest output, or, for the dark part of a picture, of that part's."""
import numpy as np
import pytest

from bm3d_b200 import core, source, synth

pytestmark = pytest.mark.gpu

REL = 2e-5
SCALES = [1e-30, 1e-15, 1e-7, 1e-6, 1e-4, 1e-2, 1.0, 255.0, 1e6, 1e15]


def run(orc, img, profile, sigma, **over):
    img = np.ascontiguousarray(img, np.float32)
    got = core.bm3d.Basic(source(img, "GRAY" if img.shape[1] == 1 else "YUV"), profile=profile, sigma=sigma, matrix=6, **over).numpy()
    p = orc.default_params(0, False, profile, sigma, matrix=6, **over)
    return got, orc.bm3d(p, img, threads=8)


@pytest.mark.parametrize("scale", SCALES)
@pytest.mark.parametrize("profile,G", [("fast", 8), ("np", 16), ("np", 32)])
@pytest.mark.parametrize("sigma", [10.0, 1.0])
def test_scaled_clip(orc, scale, profile, G, sigma):
    """sigma 1: most coefficients are kept, so the terms are smallest against the pixels."""
    nz = synth.gray_frames(5, 1, 62, 87, 10.0)[0] * np.float64(scale)
    got, exp = run(orc, nz, profile, sigma * scale, group_size=G, th_mse=2000.0 * scale * scale)
    assert np.abs(got - exp).max() <= REL * np.abs(exp).max()


@pytest.mark.parametrize("dark", [1e-2, 1e-4, 1e-6])
def test_dark_part_of_a_bright_picture(orc, dark):
    """The tile's scale follows its bright part; the dark part keeps its own precision."""
    nz = synth.gray_frames(7, 1, 48, 96, 10.0)[0]
    nz[..., 40:] *= np.float32(dark)
    got, exp = run(orc, nz, "np", 10.0 * dark, th_mse=2000.0 * dark * dark)
    assert np.abs(got - exp).max() <= REL * np.abs(exp).max()
    part = np.s_[..., 48:]                                  # blocks that start at column 40 or later
    assert np.abs(got - exp)[part].max() <= REL * np.abs(exp[part]).max()


def test_planes_of_different_magnitude(orc):
    """Chroma around zero and far smaller than luma, groups of all lengths."""
    nz = np.concatenate([synth.gray_frames(9 + k, 1, 56, 80, 10.0)[0] for k in range(3)], axis=1)
    nz[:, 1] = (nz[:, 1] - 0.5) * np.float32(1e-5)
    nz[:, 2] = 0.0
    got, exp = run(orc, nz, "np", [10.0, 1e-4, 10.0], th_mse=250.0)
    for p in range(3):
        assert np.abs(got[:, p] - exp[:, p]).max() <= REL * np.abs(exp[:, p]).max()
