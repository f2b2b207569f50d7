"""Plain Basic and Final filters on either side of the rules that choose between a tile's box in shared memory and
warp pairs on the planes: search windows with few candidates, and boxes that hold too few groups.  Against the oracle.

Tolerance: both sides run the same transforms; they differ in the order of the sums of a pixel's terms.  A pixel takes
at most 2^12 terms: rounding errors being independent, within 2^6 * 2^-24 = 4e-6 of the value range; the bound used is
2e-5."""
import numpy as np
import pytest

from bm3d_b200 import core, source, synth

pytestmark = pytest.mark.gpu

REL = 2e-5


@pytest.mark.parametrize("wiener", [0, 1])
@pytest.mark.parametrize("R,step,G", [
    (1, 8, 8), (2, 4, 8), (3, 4, 8),                        # 9, 25 and 49 candidates against 4 G = 32
    (3, 4, 16), (4, 4, 16),                                 # 49, 81 against 64
    (5, 4, 32), (6, 4, 32),                                 # 121, 169 against 128
    (9, 8, 8), (12, 8, 8), (15, 8, 8), (18, 8, 8),          # boxes of many groups, a few, one slot, none
    (16, 8, 16), (18, 8, 16), (20, 4, 16), (24, 4, 16), (26, 4, 16),
    (20, 3, 32), (22, 3, 32), (24, 8, 32), (28, 3, 32),
])
def test_forms(orc, wiener, R, step, G):
    nz, clean = synth.gray_frames(31, 1, 83, 118, 10.0)
    ref = (clean + np.random.default_rng(4).normal(0, 0.006, clean.shape)).astype(np.float32)
    over = dict(bm_range=R, block_step=step, group_size=G)
    if wiener:
        got = core.bm3d.Final(source(nz, "GRAY"), source(ref, "GRAY"), profile="np", matrix=6, **over).numpy()
    else:
        got = core.bm3d.Basic(source(nz, "GRAY"), profile="np", matrix=6, **over).numpy()
    p = orc.default_params(wiener, False, "np", 10.0, matrix=6, **over)
    exp = orc.bm3d(p, nz, ref if wiener else None, threads=8)
    assert np.abs(got - exp).max() <= REL * max(1.0, np.abs(exp).max())
