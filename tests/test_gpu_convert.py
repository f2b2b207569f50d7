"""Conversions, bit for bit against the oracle: eight samples a thread with 16-byte accesses and the scalar form,
row remainders, planes off their alignment, and more frames than one launch takes."""
import numpy as np
import pytest

from bm3d_b200 import core, source

pytestmark = pytest.mark.gpu


def view(a, pad, shift):
    """The array on the GPU with `pad` extra columns per row, starting `shift` samples into its buffer."""
    import torch
    n, p, h, w = a.shape
    buf = torch.zeros(n * p * h * (w + pad) + shift, dtype=getattr(torch, str(a.dtype)), device="cuda")
    v = buf[shift:].view(n, p, h, w + pad)[..., :w]
    v.copy_(torch.from_numpy(a).cuda())
    return v


@pytest.mark.parametrize("dtype,bits", [(np.uint8, 8), (np.uint16, 16), (np.float32, 32)])
@pytest.mark.parametrize("h,w,frames,pad,shift", [
    (3, 8, 1, 0, 0), (5, 64, 2, 0, 0), (4, 61, 1, 3, 0), (7, 13, 1, 0, 0), (2, 1, 1, 0, 0), (6, 72, 1, 8, 1), (4, 40, 19, 0, 0),
])
def test_rgb_opp_rgb(orc, dtype, bits, h, w, frames, pad, shift):
    rng = np.random.default_rng(h * 100 + w)
    rgb = rng.random((frames, 3, h, w))
    rgb = rgb.astype(np.float32) if bits == 32 else np.round(rgb * ((1 << bits) - 1)).astype(dtype)
    src = source(view(rgb, pad, shift), "RGB")
    for sample, out in ((1, np.float32), (0, np.uint16)):
        opp = core.bm3d.RGB2OPP(src, sample=sample)
        exp = np.stack([orc.rgb2opp_any(f, out) for f in rgb])
        got = np.stack([f.numpy() for f in opp.get_frames(0, frames)])
        assert np.array_equal(got, exp)
        back = core.bm3d.OPP2RGB(opp, sample=sample)
        got = np.stack([f.numpy() for f in back.get_frames(0, frames)])
        assert np.array_equal(got, np.stack([orc.opp2rgb_any(f, out) for f in exp]))


@pytest.mark.parametrize("w,shift", [(64, 0), (61, 0), (64, 3)])
def test_unprocessed_planes_are_copied(w, shift):
    rng = np.random.default_rng(w)
    yuv = np.round(rng.random((2, 3, 16, w)) * 65535).astype(np.uint16)
    out = core.bm3d.Basic(source(view(yuv, 0, shift), "YUV"), sigma=[0.0, 0.0, 0.0])
    assert np.array_equal(np.stack([f.numpy() for f in out.get_frames(0, 2)]), yuv)
