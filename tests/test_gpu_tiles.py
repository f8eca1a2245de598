"""The tile gather (GatherData) where its marches skip: grids that are and are
not powers of two, nonzero boxes off the centre, of one voxel and none, steps
bounded by the majorant, an odd tile grid; against the CPU oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_scene import LIGHT, view_frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alpha", [4.0, 900.0])
@pytest.mark.parametrize("R,lo,hi,storage", [(64, (0, 0, 0), (64, 64, 64), "fp32"), (48, (20, 3, 17), (40, 25, 30), "fp16"),
                                             (37, (30, 20, 10), (31, 21, 11), "fp32"), (32, (0, 0, 0), (0, 0, 0), "fp32"),
                                             (32, (8, 8, 8), (24, 24, 24), "fp16")])
def test_tiles(alpha, R, lo, hi, storage):
    """The float order is the reference's, so marches and samples agree with
    the oracle up to the logarithms' and exponentials' last bits (the bar of
    the existing tile test); a value may differ more where such a bit decides
    a step, which the share allows for."""
    import mrpnn_b200 as M
    M.init()
    rng = np.random.default_rng(R)
    data = np.zeros((R, R, R), np.float32)
    data[lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]] = rng.uniform(0.0, 1.0, [h - l for l, h in zip(lo, hi)])
    if storage == "fp16":
        data = data.astype(np.float16).astype(np.float32)
    v = M.VolumeRender(R, storage=storage)
    v.set_data(data)
    v.Update()
    v.UpdateHGLut(0.857)
    v.Update_TR(LIGHT, alpha)
    ori, up, right = view_frame()
    W, H = 11, 7
    got = v.GatherData((W, H), ori, up, right, LIGHT, alpha=alpha, g=0.857, pixelOffset=(1, 6), seed=3)
    mips = np.concatenate([v.read(M.api.RES_MIP, m) for m in range(9)])
    trs = np.concatenate([v.read(M.api.RES_TR, m) for m in range(8)])
    sc = O.SceneBuf(data.ravel(), R, v.max_density, mips, trs, v.read(M.api.RES_LUT))
    ref = O.gather_tiles(sc, O.make_view(W, H, ori, up, right, LIGHT, alpha=alpha, g=0.857, seed=3, frame=0), 1, 6)
    assert np.array_equal(got[:, 0] == -1000.0, ref[:, 0] == -1000.0)
    ok = np.isclose(got, ref, rtol=1e-4, atol=1e-5)
    assert ok.mean() > 0.999, (ok.mean(), np.abs(got - ref).max())
