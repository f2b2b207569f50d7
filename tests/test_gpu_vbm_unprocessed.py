"""V-BM3D with every sigma zero: no plane is processed, and the request is answered like one whose unprocessed planes
are left alone -- the aggregated output of such planes is zero, the stacked clip says that none was processed."""
import numpy as np
import pytest

from bm3d_b200 import core, source

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family,planes", [("GRAY", 1), ("YUV", 3)])
@pytest.mark.parametrize("sample", [0, 1])
@pytest.mark.parametrize("func", ["VBasic", "VFinal"])
def test_no_plane_processed(family, planes, sample, func):
    src = source(np.random.default_rng(0).random((3, planes, 24, 33)).astype(np.float32), family)
    clips = (src, src) if func == "VFinal" else (src,)
    make = getattr(core.bm3d, func)
    out = make(*clips, sigma=[0.0, 0.0, 0.0], radius=1, aggregate=1, sample=sample).get_frames(0, 3)
    assert all(not f.numpy().any() for f in out)
    stacked = make(*clips, sigma=[0.0, 0.0, 0.0], radius=1).get_frames(0, 3)
    for f in stacked:
        assert not any(f.props["BM3D_V_process"])
        assert f.numpy().shape == (planes, 24 * 6, 33)
