"""The stencil gather splits a record's points over six threads for small
launches; the tensor-core forms do not above 600 000 pixels.  A ray's radiance
does not depend on it: the first rays of a launch on either side of the line
give the same bits."""
import numpy as np
import pytest

from tests.gpu_scene import LIGHT, Scene, view_frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,hardware", [(1, True), (1, False), (2, True), (0, False)])
def test_parts_do_not_show(precision, hardware):
    import mrpnn_b200 as M
    sc = Scene(R=64)
    v = sc.vol
    v.SetPrecision(precision)
    v.SetGatherFilter(hardware)
    ori, up, right = view_frame()
    rng = np.random.default_rng(7)
    fwd = -ori / np.linalg.norm(ori)
    d = fwd + rng.uniform(-1, 1, (600001, 1)) * right + rng.uniform(-1, 1, (600001, 1)) * up
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)

    def radiances(n):
        return v.GetRadiances(np.broadcast_to(ori, (n, 3)), d[:n], LIGHT, (1, 1, 1), sc.alpha, 1, sc.g, 1,
                              M.VolumeRender.MRPNN)

    whole = radiances(600001)
    assert (whole.sum(1) > 0.2).mean() > 0.3   # a good part of the rays hit the cloud
    for n in (1, 127, 129, 1000):
        np.testing.assert_array_equal(radiances(n), whole[:n])
