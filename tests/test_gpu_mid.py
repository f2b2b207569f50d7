"""Filter of small groups of blocks other than the 8 x 8 box form, against the oracle: every class of block size
(unrolled, direct with 4 / 8 / 12 / 16 outputs side by side), group lengths, one size beyond it on either side,
and V-BM3D.

Tolerance: the transforms are the oracle's, operation for operation; the sums of a pixel's terms and, for
Final, of the squared weights run in another order.  At most 2^13 terms of one sign each: rounding errors
being independent, within 2^6.5 * 2^-24 = 6e-6 of the value range; the bound used is 2e-5."""
import numpy as np
import pytest

from bm3d_b200 import core, source, synth

pytestmark = pytest.mark.gpu

REL = 2e-5


@pytest.mark.parametrize("wiener", [0, 1])
@pytest.mark.parametrize("over", [
    {"block_size": 2, "block_step": 2}, {"block_size": 3, "block_step": 2}, {"block_size": 4, "block_step": 3},
    {"block_size": 5, "block_step": 3}, {"block_size": 7, "block_step": 4}, {"block_size": 9, "block_step": 5},
    {"block_size": 11, "block_step": 6}, {"block_size": 12, "block_step": 6}, {"block_size": 13, "block_step": 7},
    {"block_size": 16, "block_step": 8}, {"block_size": 17, "block_step": 8},
    {"group_size": 1}, {"group_size": 12}, {"group_size": 27}, {"group_size": 33},
    {"block_size": 11, "block_step": 6, "th_mse": 40.0},
])
def test_mid_filter_matches_oracle(orc, wiener, over):
    over = dict({"bm_range": 9, "block_step": 4, "group_size": 32}, **over)
    if "th_mse" in over and not wiener:
        over["th_mse"] = 300.0
    nz, clean = synth.gray_frames(21, 2, 45, 58, 10.0)
    ref = (clean + np.random.default_rng(2).normal(0, 0.006, clean.shape)).astype(np.float32)
    if wiener:
        got = core.bm3d.Final(source(nz, "GRAY"), source(ref, "GRAY"), profile="np", matrix=6, **over).numpy()
    else:
        got = core.bm3d.Basic(source(nz, "GRAY"), profile="np", matrix=6, **over).numpy()
    p = orc.default_params(wiener, False, "np", 10.0, matrix=6, **over)
    exp = orc.bm3d(p, nz, ref if wiener else None, threads=8)
    assert np.abs(got - exp).max() <= REL


@pytest.mark.parametrize("B", [5, 16])
def test_mid_filter_video(orc, B):
    nz, _ = synth.motion_frames(3, 3, 40, 48, 12.0, planes=1)
    nz = nz.astype(np.float32)
    over = dict(block_size=B, block_step=4, radius=1)
    got = core.bm3d.VBasic(source(nz, "GRAY"), matrix=6, **over).numpy()
    p = orc.default_params(0, True, "fast", 10.0, matrix=6, **over)
    exp = orc.vbm3d(p, nz)
    # stacked numerators and weights: sums of up to 2^13 weighted terms, compared on their own scale
    assert np.abs(got - exp).max() <= REL * np.abs(exp).max()
