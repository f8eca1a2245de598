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


@pytest.mark.parametrize("g", [0.3, 0.857])
@pytest.mark.parametrize("sign", [1, -1])
def test_phase_rows_at_the_ends(sign, g):
    """The phase features with the light along the view, whose cosines lie at
    the ends of the points' rows of the phase table.  A cosine differs from the
    oracle's by a few ulp, 2e-7, which is 5e-5 of a texel; neighbouring texels
    of the cone-averaged table differ by less than a factor of 2, two factors:
    1e-4, and once more for their blend's rounding."""
    from oracle import oracle as O
    sc = Scene(R=64, g=g)
    W = 32
    ori, up, right = view_frame()
    light = (sign * ori / np.linalg.norm(ori)).astype(np.float32)
    _, aux, feat = sc.vol.predict_debug(sc.vol.make_view((W, W), ori, up, right, light, g, sc.alpha, seed=3))
    view = O.make_view(W, W, ori, up, right, light, alpha=sc.alpha, g=g, seed=3, frame=0)
    _, ref, _, hits = O.predict_pixels(sc.orc, view, np.arange(W * W, dtype=np.int32), want_features=True)
    hit = hits[:, 3] > 0
    assert hit.sum() > 100
    np.testing.assert_array_equal(aux[:, 3] > 0, hit)
    np.testing.assert_allclose(feat[hit, 384:], ref[hit, 384:], rtol=2e-4, atol=1e-6)


@pytest.mark.parametrize("W,H", [(37, 23), (163, 149), (201, 190)])
def test_march_tiles(W, H):
    """8, 16 and 32 pixels a warp, over images that their tiles do not divide:
    pixels all over the frame, its last rows and columns among them, against the
    oracle to the FP32 predictor's bound."""
    import mrpnn_b200 as M
    from oracle import oracle as O
    sc = Scene(R=64)
    ori, up, right = view_frame()
    got = sc.vol.Render((W, H), ori, up, right, LIGHT, M.VolumeRender.MRPNN, sc.g, sc.alpha, sampleNum=1,
                        seed=3).reshape(-1, 4)
    yx = np.random.default_rng(W).integers(0, (H, W), (300, 2))
    yx[:40, 0] = H - 1 - np.arange(40) % 2
    yx[40:80, 1] = W - 1 - np.arange(40) % 2
    pix = np.unique(yx[:, 0] * W + yx[:, 1]).astype(np.int32)
    view = O.make_view(W, H, ori, up, right, LIGHT, alpha=sc.alpha, g=sc.g, seed=3, frame=0)
    ref = O.predict_pixels(sc.orc, view, pix)
    assert (ref[:, 3] > 0).sum() > 50
    np.testing.assert_allclose(got[pix], ref, rtol=1e-4, atol=1e-6)


@pytest.mark.parametrize("precision,hardware", [(1, True), (1, False), (0, False)])
def test_six_and_twelve_parts(precision, hardware):
    """Launches on either side of the line between six and twelve threads a
    record: the same rays, the same bits."""
    import torch

    import mrpnn_b200 as M
    sc = Scene(R=64)
    sc.vol.SetPrecision(precision)
    sc.vol.SetGatherFilter(hardware)
    ori, up, right = view_frame()
    n = 512 * torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(8)
    d = -ori / np.linalg.norm(ori) + rng.uniform(-1, 1, (n + 1, 1)) * right + rng.uniform(-1, 1, (n + 1, 1)) * up
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)

    def radiances(k):
        return sc.vol.GetRadiances(np.broadcast_to(ori, (k, 3)), d[:k], LIGHT, (1, 1, 1), sc.alpha, 1, sc.g, 1,
                                   M.VolumeRender.MRPNN)

    np.testing.assert_array_equal(radiances(n), radiances(n + 1)[:n])


@pytest.mark.parametrize("precision,hardware", [(1, True), (1, False), (2, False), (0, False)])
def test_hits_at_infinity(precision, hardware):
    """A density of -infinity takes a march to an infinite position, the hit
    the reference's arithmetic gives there; the gathers read no texel for it
    (a coordinate made of it is the largest integer).  Hits as the oracle's:
    the march's order is the reference's up to the last bits of a logarithm."""
    import mrpnn_b200 as M
    from oracle import oracle as O
    M.init()
    R, W, H = 5, 33, 18
    data = np.random.default_rng(3).uniform(0.05, 3.0, (R, R, R)).astype(np.float32)
    data.ravel()[13] = -np.inf
    v = M.VolumeRender(R)
    v.set_data(data)
    v.Update()
    v.SetPrecision(precision)
    v.SetGatherFilter(hardware)
    ori, up, right = view_frame()
    view = v.make_view((W, H), ori, up, right, LIGHT, 0.857, 64.0, seed=8)
    rgba, aux, _ = v.predict_debug(view)
    mips = np.concatenate([v.read(M.api.RES_MIP, m) for m in range(9)])
    sc = O.SceneBuf(data.ravel(), R, v.max_density, mips, np.concatenate([v.read(M.api.RES_TR, m) for m in range(8)]),
                    v.read(M.api.RES_LUT))
    ov = O.make_view(W, H, ori, up, right, LIGHT, alpha=64.0, g=0.857, seed=8, frame=0)
    _, _, _, hits = O.predict_pixels(sc, ov, np.arange(W * H, dtype=np.int32), want_features=True)
    hit = hits[:, 3] > 0
    assert np.isinf(hits[hit, :3]).any() and np.isfinite(hits[hit, :3]).all(1).sum() > 20
    np.testing.assert_array_equal(aux[:, 3] > 0, hit)
    np.testing.assert_allclose(aux[hit, :3], hits[hit, :3], rtol=1e-5, atol=1e-6)
    frame = v.Render((W, H), ori, up, right, LIGHT, v.MRPNN, 0.857, 64.0, sampleNum=1, seed=8)
    np.testing.assert_array_equal(frame.reshape(-1, 4), rgba)


def test_features_far_away():
    """Points beyond any integer texel coordinate: no density, and no shadow
    where the light ray misses the box."""
    sc = Scene(R=64)
    far = [1e12, 1e30, 1e35, float("inf")]
    pos = np.zeros((3 * len(far), 3), np.float32)
    for a in range(3):
        pos[a * len(far):(a + 1) * len(far), a] = far
    frame = np.tile(np.array([1, 0, 0, 0, 1, 0, 0, 0, 1, *LIGHT], np.float32), (len(pos), 1))
    feat, _ = sc.vol.gather_features(pos, frame, np.abs(LIGHT), sc.g, sc.alpha)
    finite = np.isfinite(pos).all(1)
    np.testing.assert_array_equal(feat[finite, :192], 0.0)
    np.testing.assert_array_equal(feat[finite, 192:384], 1.0)
