"""Plain Basic and Final filters with the image region of a tile in shared memory, against the oracle: tile and
slot edges, every kind of group length, block (0, 0) inside and outside the box, terms too large for
the fixed-point box, NaN, and search ranges at and beyond the largest box.

Tolerance: both sides run the same transforms; they differ in the order of the sums of a pixel's
terms.  A pixel takes at most 2^12 terms, so the oracle's sequential fp32 sums are within
2^12 * 2^-24 = 2.4e-4 of its largest partial sum in the worst case and, rounding errors being
independent, within 2^6 * 2^-24 = 4e-6 in practice; the bound used is 2e-5 of the value range."""
import numpy as np
import pytest

from bm3d_b200 import core, source, synth

pytestmark = pytest.mark.gpu

REL = 2e-5


def pair(h, w, sigma=10.0, seed=3):
    nz, clean = synth.gray_frames(seed, 1, h, w, sigma)
    ref = clean + np.random.default_rng(seed).normal(0, 0.15 * sigma / 255.0, clean.shape)
    return nz, ref.astype(np.float32)


def check(orc, src, ref, profile="np", **over):
    """ref None: Basic of src"""
    if ref is None:
        node = core.bm3d.Basic(source(src, "GRAY"), profile=profile, matrix=6, **over)
    else:
        node = core.bm3d.Final(source(src, "GRAY"), source(ref, "GRAY"), profile=profile, matrix=6, **over)
    got = node.numpy()
    p = orc.default_params(0 if ref is None else 1, False, profile, 10.0, matrix=6, **over)
    exp = orc.bm3d(p, src, ref, threads=8)
    assert np.array_equal(np.isnan(got), np.isnan(exp))
    ok = ~np.isnan(exp)
    scale = max(1.0, float(np.abs(exp[ok]).max()))
    assert np.abs(got - exp)[ok].max() <= REL * scale


CASES = [
    (8, 8, {}),                                                  # one block: one group of one
    (9, 47, {}),                                                 # window taller than the frame
    (41, 13, {}),                                                # window wider than the frame
    (67, 131, {}),                                               # several tiles, ragged last ones
    (70, 133, {"group_size": 8}),                                # four groups per slot
    (70, 133, {"group_size": 16}),                               # two
    (64, 96, {"th_mse": 12.0}),                                  # mostly short groups, any length
    (64, 96, {"group_size": 16, "th_mse": 12.0}),
    (64, 96, {"group_size": 8, "th_mse": 12.0}),
    (72, 200, {"block_step": 8, "bm_range": 4}),                 # tiles far wider than the window
    (60, 90, {"block_step": 1}),
    (120, 140, {"bm_range": 36}),                                # one CTA per SM
    (200, 230, {"bm_range": 60, "block_step": 8}),               # beyond any box: per-lane kernel
    (64, 80, {"bm_range": 6, "bm_step": 4}),                     # range rounded down to the step
]


@pytest.mark.parametrize("h,w,over", CASES)
def test_final_matches_oracle(orc, h, w, over):
    check(orc, *pair(h, w), **over)


@pytest.mark.parametrize("h,w,over", CASES)
def test_basic_matches_oracle(orc, h, w, over):
    """Two slots at a time: odd numbers of slots and of groups in them, and groups of different lengths."""
    if "th_mse" in over:
        over = dict(over, th_mse=300.0)                          # noisy blocks: short groups below it
    check(orc, pair(h, w)[0], None, **over)


def test_block_at_origin_in_distant_groups(orc):
    """Flat pictures: the trailing candidate (0, 0) of the search list joins groups of every tile."""
    rng = np.random.default_rng(9)
    src = (0.5 + 0.04 * rng.normal(size=(1, 1, 80, 160))).astype(np.float32)
    ref = (0.5 + 0.01 * rng.normal(size=(1, 1, 80, 160))).astype(np.float32)
    ref[..., :8, :8] = 0.5 + 0.2 * (ref[..., :8, :8] - 0.5)
    check(orc, src, ref)


def test_terms_beyond_the_fixed_point_box(orc):
    src, ref = pair(56, 72)
    check(orc, src * np.float32(1e6), ref * np.float32(1e6), th_mse=1e15)
    check(orc, src * np.float32(1e6), None, th_mse=1e15)


def test_nan_stays_in_the_groups_that_hold_it(orc):
    src, ref = pair(64, 96)
    src[0, 0, 30, 40] = np.nan
    check(orc, src, ref, th_mse=40.0)
    check(orc, src, None)


def test_weights_of_huge_values(orc):
    """Spectra whose squares leave the range of the reciprocal estimate (and, further on, of fp32)."""
    src, ref = pair(40, 56)
    check(orc, src * np.float32(1e15), ref * np.float32(1e15), th_mse=1e33)
