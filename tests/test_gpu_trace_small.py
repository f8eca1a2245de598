"""The tracer's event loop where its batches do not fill: fewer samples than
lanes, one bounce, rays that miss, one sample a pixel; per pixel against the
oracle, whose paths take the same draws."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_scene import LIGHT, Scene, view_frame

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene():
    return Scene(R=40, bake_res=32)


@pytest.mark.parametrize("w,h,spp,bounces", [(1, 1, 1, 64), (5, 3, 1, 1), (31, 1, 3, 64), (33, 2, 2, 2), (40, 37, 1, 64),
                                             (64, 64, 5, 256)])
def test_small_images(scene, w, h, spp, bounces):
    """The frame's free flight takes the fast log and division (4e-7 of a mean
    free path), so a step's accept test falls the other way where a draw lies
    within about 1e-6 of it: with some fifty steps a sample, one sample in
    10 000; 3 % of the pixels is far above that for 5 samples each.  Samples on
    the same path agree to the positions' rounding, far below 1e-3."""
    ori, up, right = view_frame()
    got = scene.vol.Render((w, h), ori, up, right, LIGHT, scene.vol.PT, scene.g, scene.alpha, multiScatter=bounces,
                           sampleNum=1, spp=spp, seed=9).reshape(-1, 4)
    view = O.make_view(w, h, ori, up, right, LIGHT, alpha=scene.alpha, g=scene.g, multi_scatter=bounces, spp=spp, seed=9,
                       frame=0)
    ref = O.trace_pixels(scene.orc, view, np.arange(w * h, dtype=np.int32))[0][:, :3]
    bad = (np.abs(got[:, :3] - ref) > 1e-3 * np.maximum(np.abs(ref), 1e-3)).any(axis=1)
    assert bad.mean() <= 0.03
